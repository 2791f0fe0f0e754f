"""What stands between a weight write and the matmul behind it on the same stream, and between chained prefill launches.

The matmul kernels read weights before they wait for the kernel in front of them, so a call straight behind a repack must be a
fully ordered launch, whatever was refused in between, and any other call may be a programmatic one. The kind of ordering
is read from captured graphs; the results are compared bit for bit with runs that synchronise after every call."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

FULL, PROGRAMMATIC = 0, 1  # CUgraphDependencyType


class _EdgeData(C.Structure):
    _fields_ = [("from_port", C.c_ubyte), ("to_port", C.c_ubyte), ("type", C.c_ubyte), ("reserved", C.c_ubyte * 5)]


def _edges(fn):
    """Edge kinds, first to last, of the chain of nodes that `fn(stream)` captures."""
    cuda = C.CDLL("libcuda.so.1")
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        fn(stream)
    handle, n = C.c_void_p(graph.raw_cuda_graph()), C.c_size_t(0)
    assert cuda.cuGraphGetEdges_v2(handle, None, None, None, C.byref(n)) == 0
    src, dst, data = (C.c_void_p * n.value)(), (C.c_void_p * n.value)(), (_EdgeData * n.value)()
    assert cuda.cuGraphGetEdges_v2(handle, src, dst, data, C.byref(n)) == 0
    nxt = {src[i]: (dst[i], data[i].type) for i in range(n.value)}
    assert len(nxt) == n.value, "not a chain"
    node, kinds = next(iter(set(nxt) - {d for d, _ in nxt.values()})), []
    while node in nxt:
        node, kind = nxt[node]
        kinds.append(kind)
    return kinds


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
    assert _edges(chain) == [PROGRAMMATIC] * (n - 1) + [FULL, FULL] + [PROGRAMMATIC] * (2 * n - 1)


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

    assert _edges(chain) == [FULL] + [PROGRAMMATIC] * (n - 1)
