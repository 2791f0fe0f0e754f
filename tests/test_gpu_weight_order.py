"""What stands between a weight write and the matmul behind it on the same stream, and between chained prefill launches.

The matmul kernels read weights before they wait for the kernel in front of them, so a call straight behind a repack must be a
fully ordered launch, whatever was refused in between, and any other call may be a programmatic one. The kind of ordering
is read from captured graphs; the results are compared bit for bit with runs that synchronise after every call."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from gpu_util import captured_edges  # noqa: E402

pytestmark = pytest.mark.gpu

FULL, PROGRAMMATIC = 0, 1  # CUgraphDependencyType


def _tensors(synth, N, K, seed):
    packed, scale, zp = synth.make_weights(N, K, seed=seed)
    return (torch.from_numpy(packed.view(np.int32)).cuda(), torch.from_numpy(scale.view(np.int16)).cuda(),
            torch.from_numpy(zp.view(np.int32)).cuda())


@pytest.fixture(scope="module")
def layer(pkg, synth):
    N = K = 1024
    src = _tensors(synth, N, K, 1)
    w = pkg.awq_repack(*src)
    narrow, wide = pkg.gemv_scratch_alloc(K, 128, 128, 1), pkg.gemv_scratch_alloc(K, N, 128, 1)
    block, ws = pkg.gemv_scratch_alloc(K, N, 128, 16), pkg.gemm_workspace_alloc(4096)
    gen = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn((80, K), device="cuda", generator=gen).to(torch.bfloat16)
    y = torch.empty((80, N), dtype=torch.bfloat16, device="cuda")
    calls = {  # matmuls that run, by name, and the number of kernels of each
        "gemv": (lambda st: pkg.gemv_w4a16(y, w, x, wide, stream=st), 1),
        "skinny": (lambda st: pkg.gemm_small_w4a16(y, w, x, 9, block, stream=st), 2),
        "prefill": (lambda st: pkg.gemm_w4a16(y, w, x, 77, ws, stream=st), 1),
    }
    odd = x.view(-1)[1:]
    refused = {
        "scratch too small for the rows": lambda st: pkg.gemv_w4a16(y, w, x, narrow, stream=st),
        "scratch too small for the tokens": lambda st: pkg.gemm_small_w4a16(y, w, x, 2, wide, stream=st),
        "norm without room": lambda st: pkg.linear_fused(y, w, x, 1, wide, ln_weight=x[1], stream=st),
        "prefill off alignment": lambda st: pkg.gemm_w4a16(y, w, odd, 70, ws, stream=st),
    }
    for fn, _ in calls.values():  # one-time set-up of the kernels, before any capture
        fn(torch.cuda.current_stream())
    torch.cuda.synchronize()
    yield src, w, calls, refused
    assert pkg.device_status() == 0
    for s in (narrow, wide, block):
        pkg.gemv_scratch_free(s)
    pkg.gemm_workspace_free(ws)
    pkg.awq_free(w)


@pytest.mark.parametrize("name", ["gemv", "skinny", "prefill"])
def test_first_matmul_behind_a_repack_is_fully_ordered(pkg, layer, name):
    src, w, calls, _ = layer
    fn, n = calls[name]

    def chain(st):
        fn(st)
        pkg.awq_repack_into(w, 0, *src, stream=st)
        fn(st)
        fn(st)

    # inside the first call, into the repack, into the call behind it, and from there on
    assert captured_edges(chain) == [PROGRAMMATIC] * (n - 1) + [FULL, FULL] + [PROGRAMMATIC] * (2 * n - 1)


@pytest.mark.parametrize("name", ["gemv", "skinny", "prefill"])
@pytest.mark.parametrize("why", ["scratch too small for the rows", "scratch too small for the tokens", "norm without room",
                                 "prefill off alignment"])
def test_refused_call_leaves_the_ordering_to_the_next(pkg, layer, name, why):
    src, w, calls, refused = layer
    fn, n = calls[name]

    def chain(st):
        pkg.awq_repack_into(w, 0, *src, stream=st)
        with pytest.raises(pkg.W4A16Error):
            refused[why](st)
        fn(st)

    assert captured_edges(chain) == [FULL] + [PROGRAMMATIC] * (n - 1)


@pytest.mark.parametrize("name", ["gemv", "skinny", "prefill"])
def test_captured_calls_leave_the_ordering_to_the_next_executed_one(pkg, layer, name):
    """What a later call would get is read from a capture, of which only the edges count: the first matmul behind the write is
    fully ordered in every capture, however many there are, until a call on the stream has been executed."""
    src, w, calls, _ = layer
    fn, n = calls[name]
    stream, rows = torch.cuda.Stream(), torch.empty((w.out_f, w.in_f), dtype=torch.bfloat16, device="cuda")

    def chain(st):
        pkg.w4a16_dequant_rows(rows, w, 0, w.out_f, stream=st)  # the node in front of the first matmul
        fn(st)
        fn(st)

    ordered, free = [FULL] + [PROGRAMMATIC] * (2 * n - 1), [PROGRAMMATIC] * (2 * n)
    assert captured_edges(chain, stream) == free
    pkg.awq_repack_into(w, 0, *src, stream=stream)
    assert captured_edges(chain, stream) == ordered
    assert captured_edges(chain, stream) == ordered
    fn(stream)
    assert captured_edges(chain, stream) == free
    # a write that is captured itself: the matmul behind it, and the next executed one
    assert captured_edges(lambda st: (pkg.awq_repack_into(w, 0, *src, stream=st), chain(st)), stream) == [FULL] + ordered
    fn(stream)
    assert captured_edges(chain, stream) == free
    torch.cuda.synchronize()


@pytest.mark.parametrize("name", ["gemv", "skinny", "prefill"])
def test_executed_call_behind_a_repack_and_a_capture(pkg, synth, layer, name):
    """Repack, a matmul that is only captured, the same matmul executed: the new weights' bits."""
    src, w, calls, _ = layer
    other = _tensors(synth, w.out_f, w.in_f, 9)
    stream = torch.cuda.Stream()
    x = torch.randn((80, w.in_f), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).to(torch.bfloat16)
    y = [torch.zeros((80, w.out_f), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    block, ws = pkg.gemv_scratch_alloc(w.in_f, w.out_f, 128, 16), pkg.gemm_workspace_alloc(4096)
    call = {"gemv": lambda out: pkg.gemv_w4a16(out, w, x, block, stream=stream),
            "skinny": lambda out: pkg.gemm_small_w4a16(out, w, x, 9, block, stream=stream),
            "prefill": lambda out: pkg.gemm_w4a16(out, w, x, 77, ws, stream=stream)}[name]
    torch.cuda.synchronize()
    for tensors in (other, src) * 4:
        call(y[0])  # the old weights' call in front
        pkg.awq_repack_into(w, 0, *tensors, stream=stream)
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=stream):
            call(y[1])
        call(y[0])
        torch.cuda.synchronize()
        call(y[1])
        torch.cuda.synchronize()
        assert torch.equal(y[0].view(torch.int16), y[1].view(torch.int16))
    assert pkg.device_status() == 0
    pkg.gemv_scratch_free(block)
    pkg.gemm_workspace_free(ws)


def _steps(pkg, layers, ws, scratch, b, stream):
    """Prefill and decode calls in which every call reads what the one in front of it wrote, or writes what it read."""
    w0, w1, w2 = layers
    T = b["a"].shape[0]

    def prefill(dst, w, src):
        return lambda: pkg.gemm_w4a16(b[dst], w, b[src], T, ws, stream=stream)

    return [
        prefill("b", w0, "a"), prefill("c", w1, "b"), prefill("d", w2, "c"),  # C of one as A of the next
        prefill("c", w0, "d"), prefill("d", w1, "c"),                         # C over the A of the call in front
        lambda: pkg.gemm_small_w4a16(b["y"], w0, b["d"], 9, scratch, stream=stream),
        lambda: pkg.gemv_w4a16(b["d"][3], w1, b["y"][8], scratch, stream=stream),  # decode into a row that ...
        prefill("a", w2, "d"), prefill("c", w0, "a"),                         # ... the prefill behind it reads
        lambda: pkg.gemm_small_w4a16(b["a"], w1, b["c"], 16, scratch, stream=stream),
        lambda: pkg.gemv_w4a16(b["z"], w2, b["a"][15], scratch, stream=stream),
        prefill("d", w1, "a"),
    ]


# few tiles with K split over clusters and most SMs idle; more tokens; an odd number of row tiles
@pytest.mark.parametrize("H,T", [(1024, 77), (1024, 300), (640, 19), (2176, 130)])
def test_chained_prefill_and_decode_calls(pkg, synth, H, T):
    layers = [pkg.awq_repack(*_tensors(synth, H, H, 20 + i)) for i in range(3)]
    scratch, ws = pkg.gemv_scratch_alloc(H, H, 128, 16), pkg.gemm_workspace_alloc(4096)
    gen = torch.Generator(device="cuda").manual_seed(H + T)
    x = torch.randn((T, H), device="cuda", generator=gen).to(torch.bfloat16)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()

    def buffers():
        b = {n: torch.zeros((T, H), dtype=torch.bfloat16, device="cuda") for n in "abcdy"}
        b["z"] = torch.zeros(H, dtype=torch.bfloat16, device="cuda")
        b["a"].copy_(x)
        torch.cuda.synchronize()
        return b

    def same(b):
        return all(torch.equal(b[n].view(torch.int16), want[n].view(torch.int16)) for n in b)

    want = buffers()
    for step in _steps(pkg, layers, ws, scratch, want, stream):
        step()
        torch.cuda.synchronize()
    assert all(bool(torch.isfinite(t.float()).all()) for t in want.values())
    for _ in range(10):
        b = buffers()
        for step in _steps(pkg, layers, ws, scratch, b, stream):
            step()
        torch.cuda.synchronize()
        assert same(b)
    b, graph = buffers(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        b["a"].copy_(x)
        for step in _steps(pkg, layers, ws, scratch, b, stream):
            step()
    for _ in range(5):
        for n in b:
            b[n].zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert same(b)
    assert pkg.device_status() == 0
    pkg.gemv_scratch_free(scratch)
    pkg.gemm_workspace_free(ws)
    for w in layers:
        pkg.awq_free(w)


@pytest.mark.parametrize("T", [19, 300])
def test_prefill_right_behind_a_repack(pkg, synth, T):
    """The same container overwritten with new weights and multiplied at once, with no synchronisation in between."""
    H = 1024
    sources = [_tensors(synth, H, H, 30 + i) for i in range(6)]
    w, ws = pkg.awq_alloc_fused(H, H), pkg.gemm_workspace_alloc(4096)
    gen = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn((T, H), device="cuda", generator=gen).to(torch.bfloat16)
    early, settled = torch.empty_like(x), torch.empty_like(x)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for src in sources:
        pkg.gemm_w4a16(settled, w, x, T, ws, stream=stream)  # a prefill in front of the write, as well as behind it
        pkg.awq_repack_into(w, 0, *src, stream=stream)
        pkg.gemm_w4a16(early, w, x, T, ws, stream=stream)
        torch.cuda.synchronize()
        pkg.gemm_w4a16(settled, w, x, T, ws, stream=stream)
        torch.cuda.synchronize()
        assert torch.equal(early.view(torch.int16), settled.view(torch.int16))
    assert pkg.device_status() == 0
    pkg.gemm_workspace_free(ws)
    pkg.awq_free(w)
