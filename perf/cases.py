"""The work whose speed counts for this library: what a server that links it has it do, from a single small
GEMV to a prefill of 4096 tokens, through the public entry points only.

A case is a dict of plain values. `kind` says which path it takes:

  gemv     one decode GEMV (M = 1), called eagerly: the smallest unit of work a caller can ask for
  pass     the linear layers of `layers` decoder layers at M tokens, replayed as one CUDA graph, as a server
           replays its decode or verify step; every layer has its own weights
  mlp      the fused form of the MLP blocks of `layers` decoder layers (RMSNorm, gate|up with SwiGLU, down with
           the residual add), replayed as one CUDA graph
  head     lm_head with the argmax fused, logits wanted as well (sampling reads them), int4 or int8 weights
  prefill  the linear layers of one block at M prompt tokens
  load     the load-time path: tensors in the checkpoint's layout -> private layout, and back to bf16 rows

Layers are written "rows x cols" (out_f x in_f). The listed sizes are the model's own: hidden 5120, MLP 17408,
16384 / 8192 wide attention projections, 248320 vocabulary rows. Weights are int4 uniform with bf16 scales
|N(0, 0.02)| + 1e-4, activations N(0, 1) with a few outlier channels, as a residual stream has.
"""
import importlib
import math

import torch

pkg = importlib.import_module("qwen38-3090-cuda-server_b200")

GROUP = 128
HIDDEN, INTER = 5120, 17408
# the four linear layers of a decoder layer with each kind of token mixer, out_f x in_f, in execution order
MLP = ["34816x5120", "5120x17408"]
GDN = ["16384x5120", "5120x8192"] + MLP
ATTN = ["8192x5120", "5120x6144"] + MLP


def listed():
    return [
        # One attention output projection: what a caller pays for the smallest layer, launch included.
        {"name": "gemv 5120x6144", "kind": "gemv", "shape": "5120x6144", "f32": False},
        # One decode token's weight pass, all 64 layers, 12.6 GB of weights: single-stream generation.
        {"name": "decode pass", "kind": "pass", "layers": 64, "M": 1},
        # A speculative-verify block of 8 drafted tokens and one more, a quarter of the model's layers.
        {"name": "verify pass M=9", "kind": "pass", "layers": 16, "M": 9},
        # The widest block of the skinny kernel: prompts are also fed in chunks of 16.
        {"name": "verify pass M=16", "kind": "pass", "layers": 4, "M": 16},
        # The fused MLP of four layers at one token: the decode step of a server that uses the fused entry.
        {"name": "fused mlp M=1", "kind": "mlp", "layers": 4, "M": 1, "hidden": HIDDEN, "inter": INTER},
        # The vocabulary projection of a decode step and of a verify block, int4.
        {"name": "lm_head int4 M=1", "kind": "head", "bits": 4, "shape": "248320x5120", "M": 1},
        {"name": "lm_head int4 M=9", "kind": "head", "bits": 4, "shape": "248320x5120", "M": 9},
        # The same with the int8 weights, for servers that keep the head at 8 bits.
        {"name": "lm_head int8 M=9", "kind": "head", "bits": 8, "shape": "248320x5120", "M": 9},
        # Long prompts: a 4096-token chunk through the MLP.
        {"name": "prefill 4096 mlp", "kind": "prefill", "shapes": " ".join(MLP), "M": 4096},
        # The last, ragged chunk of a prompt through a whole layer.
        {"name": "prefill 777 layer", "kind": "prefill", "shapes": " ".join(GDN), "M": 777},
        # A short chat turn behind a cached prefix.
        {"name": "prefill 77 layer", "kind": "prefill", "shapes": " ".join(ATTN), "M": 77},
        # Server start: the MLP tensors of one layer into the private layout and read back for the dequant check.
        {"name": "load mlp", "kind": "load", "shapes": " ".join(MLP)},
    ]


def _log_uniform(rng, lo, hi, step):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(step, int(round(v / step)) * step)


def draw(rng):
    kind = rng.choice(["gemv", "pass", "pass", "mlp", "head", "prefill", "prefill", "load"])
    rows, cols = _log_uniform(rng, 1024, 2 * INTER, 16), _log_uniform(rng, 1024, INTER, GROUP)
    if kind == "gemv":
        return {"kind": kind, "shape": f"{rows}x{cols}", "f32": rng.random() < 0.3}
    if kind == "pass":
        M = rng.randint(1, 16)
        return {"kind": kind, "layers": _log_uniform(rng, 1, 64 if M == 1 else 16, 1), "M": M}
    if kind == "mlp":
        return {"kind": kind, "layers": rng.randint(1, 4), "M": rng.randint(1, 16),
                "hidden": _log_uniform(rng, 1024, HIDDEN, GROUP), "inter": _log_uniform(rng, 2048, INTER, GROUP)}
    if kind == "head":
        return {"kind": kind, "bits": rng.choice([4, 4, 8]), "M": rng.randint(1, 16),
                "shape": f"{_log_uniform(rng, 16384, 248320, 16)}x{_log_uniform(rng, 1024, HIDDEN, GROUP)}"}
    if kind == "prefill":
        if rng.random() < 0.5:
            shapes = rng.choice([MLP, GDN[:2], ATTN[:2]])
            return {"kind": kind, "shapes": " ".join(shapes), "M": _log_uniform(rng, 17, 4096, 1)}
        return {"kind": kind, "shapes": f"{rows}x{cols}", "M": _log_uniform(rng, 17, 4096, 1)}
    return {"kind": kind, "shapes": f"{rows}x{cols}"}


# ------------------------------------------------------------------ what a caller's program has in hand
def _shape(text):
    n, k = text.split("x")
    return int(n), int(k)


def _disk_tensors(gen, rows, cols):
    """Seeded tensors in the checkpoint's layout: packed codes, scales, packed zero points."""
    groups = cols // GROUP
    lo, hi = -2 ** 31, 2 ** 31 - 1
    packed = torch.randint(lo, hi, (rows, cols // 8), dtype=torch.int32, device="cuda", generator=gen)
    scale = (torch.randn((rows, groups), device="cuda", generator=gen).abs() * 0.02 + 1e-4).to(torch.bfloat16)
    zp = torch.randint(lo, hi, (rows // 8, groups), dtype=torch.int32, device="cuda", generator=gen)
    return packed, scale, zp


def _activations(gen, tokens, cols):
    x = torch.randn((tokens, cols), device="cuda", generator=gen)
    x[:, torch.randint(0, cols, (max(1, cols // 512),), device="cuda", generator=gen)] *= 16.0
    return x.to(torch.bfloat16)


class State:
    """Weight containers, scratch, inputs and outputs of one case; the library's allocations go back with it."""

    def __init__(self, case, seed):
        self.case = case
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.weights, self.weights8, self.scratch, self.workspace, self.graph = [], [], None, None, None

    def layer(self, rows, cols):
        w = pkg.awq_repack(*_disk_tensors(self.gen, rows, cols))
        self.weights.append(w)
        return w

    def capture(self, step):
        """One eager step (one-time set-up of the kernels), then the step as a CUDA graph."""
        self.step = step
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            step()
            stream.synchronize()
            self.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(self.graph, stream=stream):
                step()
        torch.cuda.current_stream().wait_stream(stream)

    def __del__(self):
        if torch is None or torch.cuda is None:  # the interpreter is going down, and the process's memory with it
            return
        torch.cuda.synchronize()
        self.graph = self.step = None
        for w in self.weights:
            pkg.awq_free(w)
        for w in self.weights8:
            pkg.w8a16_free(w)
        if self.scratch is not None:
            pkg.gemv_scratch_free(self.scratch)
        if self.workspace is not None:
            pkg.gemm_workspace_free(self.workspace)


def _prepare_gemv(s, case):
    rows, cols = _shape(case["shape"])
    s.w = s.layer(rows, cols)
    s.scratch = pkg.gemv_scratch_alloc(cols, rows, GROUP, 1)
    s.x = _activations(s.gen, 1, cols)
    s.y = torch.empty(rows, dtype=torch.float32 if case["f32"] else torch.bfloat16, device="cuda")


def _prepare_pass(s, case):
    M = case["M"]
    shapes = [_shape(t) for i in range(case["layers"]) for t in (ATTN if i % 4 == 3 else GDN)]
    s.scratch = pkg.gemv_scratch_alloc(INTER, 2 * INTER, GROUP, 16)
    s.y = torch.empty(sum(n for n, _ in shapes) * M, dtype=torch.bfloat16, device="cuda")
    calls, at = [], 0
    for n, k in shapes:
        calls.append((s.y[at:at + M * n], s.layer(n, k), _activations(s.gen, M, k)))
        at += M * n
    s.calls = calls

    def step():
        for y, w, x in calls:
            if M == 1:
                pkg.gemv_w4a16(y, w, x, s_scratch)
            else:
                pkg.gemm_mma_w4a16(y, w, x, M, s_scratch)

    s_scratch = s.scratch
    s.capture(step)


def _prepare_mlp(s, case):
    M, H, I = case["M"], case["hidden"], case["inter"]
    s.scratch = pkg.gemv_scratch_alloc(max(H, I), max(2 * I, H), GROUP, 16)
    blocks = []
    for _ in range(case["layers"]):
        gate_up = pkg.awq_alloc_fused(2 * I, H)
        s.weights.append(gate_up)
        for row in (0, I):
            pkg.awq_repack_into_swiglu(gate_up, row, *_disk_tensors(s.gen, I, H), I)
        norm = (torch.randn(H, device="cuda", generator=s.gen) * 0.1).to(torch.bfloat16)
        blocks.append((norm, gate_up, s.layer(H, I)))
    s.blocks = blocks
    s.h0 = _activations(s.gen, M, H)
    s.h = torch.empty_like(s.h0)
    s.act = torch.empty((M, I), dtype=torch.bfloat16, device="cuda")
    h0, h, act, scratch = s.h0, s.h, s.act, s.scratch

    def step():
        h.copy_(h0)  # the token's hidden state arrives
        for norm, gate_up, down in blocks:
            pkg.linear_fused(act, gate_up, h, M, scratch, ln_weight=norm, epilogue=pkg.EPILOGUE_SWIGLU)
            pkg.linear_fused(h, down, act, M, scratch, epilogue=pkg.EPILOGUE_RESIDUAL)

    s.capture(step)


def _prepare_head(s, case):
    rows, cols = _shape(case["shape"])
    if case["bits"] == 8:
        src = torch.randn((rows, cols), dtype=torch.bfloat16, device="cuda", generator=s.gen) * 0.02
        s.w = pkg.quantize_w8a16(src)
        s.weights8.append(s.w)
        torch.cuda.synchronize()
    else:
        s.w = s.layer(rows, cols)
    s.scratch = pkg.gemv_scratch_alloc(cols, rows, GROUP, 16)
    s.x = _activations(s.gen, case["M"], cols)
    s.logits = torch.empty((case["M"], rows), dtype=torch.bfloat16, device="cuda")
    s.ids = torch.zeros(case["M"], dtype=torch.int32, device="cuda")


def _prepare_prefill(s, case):
    s.workspace = pkg.gemm_workspace_alloc(256 << 20)
    s.calls = []
    for n, k in map(_shape, case["shapes"].split()):
        c = torch.empty((case["M"], n), dtype=torch.bfloat16, device="cuda")
        s.calls.append((c, s.layer(n, k), _activations(s.gen, case["M"], k)))


def _prepare_load(s, case):
    s.calls = []
    for n, k in map(_shape, case["shapes"].split()):
        w = pkg.awq_alloc_fused(n, k)
        s.weights.append(w)
        out = torch.empty((n, k), dtype=torch.bfloat16, device="cuda")
        s.calls.append((out, w, _disk_tensors(s.gen, n, k)))


def prepare(case, seed):
    s = State(case, seed)
    globals()["_prepare_" + case["kind"]](s, case)
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s.case["kind"]
    if kind == "gemv":
        (pkg.gemv_w4a16_f32 if s.case["f32"] else pkg.gemv_w4a16)(s.y, s.w, s.x, s.scratch)
        return s.y
    if kind == "pass":
        s.graph.replay()
        return s.y
    if kind == "mlp":
        s.graph.replay()
        return s.h, s.act
    if kind == "head":
        fn = pkg.lm_head_argmax_w8 if s.case["bits"] == 8 else pkg.lm_head_argmax
        fn(s.ids, s.w, s.x, s.case["M"], s.scratch, logits=s.logits)
        return s.ids, s.logits
    if kind == "prefill":
        for c, w, x in s.calls:
            pkg.gemm_w4a16(c, w, x, s.case["M"], s.workspace)
        return [c for c, _, _ in s.calls]
    for out, w, (packed, scale, zp) in s.calls:
        pkg.awq_repack_into(w, 0, packed, scale, zp)
        pkg.w4a16_dequant_rows(out, w, 0, out.shape[0])
    return [out for out, _, _ in s.calls]


# ------------------------------------------------------------------ what a pass cannot do without
def _weight_bytes(n, k, bits=4):
    """Codes, bf16 scales and (int4) packed zero points of one layer."""
    g = k // GROUP
    return n * k + 2 * n * g if bits == 8 else n * k // 2 + 2 * n * g + n * g // 2


def _linear(n, k, M, bits=4, out_bytes=2):
    return _weight_bytes(n, k, bits) + 2 * M * k + out_bytes * M * n, 2.0 * M * n * k


def work(case):
    kind = case["kind"]
    if kind == "load":
        # on-disk tensors in, private layout out; private layout in, bf16 rows out
        nbytes = sum(3 * _weight_bytes(n, k) + 2 * n * k for n, k in map(_shape, case["shapes"].split()))
        return {"bytes": nbytes, "flops": 0.0}
    if kind == "gemv":
        parts = [_linear(*_shape(case["shape"]), 1, out_bytes=4 if case["f32"] else 2)]
    elif kind == "pass":
        parts = [_linear(*_shape(t), case["M"]) for i in range(case["layers"]) for t in (ATTN if i % 4 == 3 else GDN)]
    elif kind == "mlp":
        M, H, I = case["M"], case["hidden"], case["inter"]
        one = (_weight_bytes(2 * I, H) + _weight_bytes(H, I) + 2 * H + 4 * M * H + 4 * M * I, 6.0 * M * H * I)
        parts = [one] * case["layers"]
    elif kind == "head":
        parts = [_linear(*_shape(case["shape"]), case["M"], bits=case["bits"])]
        parts.append((4 * case["M"], 0.0))
    else:
        parts = [_linear(*_shape(t), case["M"]) for t in case["shapes"].split()]
    return {"bytes": float(sum(b for b, _ in parts)), "flops": float(sum(f for _, f in parts))}


def tolerance(case):
    """About four times what the path differs by from the same computation in 64 bits on the same inputs."""
    kind = case["kind"]
    if kind == "load":
        return "exact"  # a bf16 weight is one rounding of an exact product: every implementation has the same bits
    if kind == "gemv" and case["f32"]:
        return {"rel": 1e-6, "max": 1e-5}  # fp32 sums: 1.2e-7 and 7e-7 on 5120x17408
    if kind == "mlp":
        return {"rel": 2e-2, "max": 0.3}  # four chained blocks, bf16 between all steps: 9e-3 and 0.1
    if kind == "prefill":
        return {"rel": 9e-3, "max": 5e-2}  # bf16 weights and outputs: 2.3e-3 and 1.3e-2
    return {"rel": 7e-3, "max": 2e-2}  # bf16 outputs: 1.7e-3 and 4e-3
