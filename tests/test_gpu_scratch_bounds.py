"""The pre-pass output of the M >= 2 decode calls stays inside the scratch the library itself asks for, at the widest in_f
that the scratch was made for."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

GUARD = 1 << 16  # bytes behind the scratch; no instance's table is longer than 256 k groups x 16 tokens x 16 bytes


def _allocation_bytes(ptr):
    """What the library asked for: the size the driver recorded for the allocation at `ptr`."""
    base, size = ctypes.c_uint64(), ctypes.c_size_t()
    cu = ctypes.CDLL("libcuda.so.1")
    assert cu.cuMemGetAddressRange_v2(ctypes.byref(base), ctypes.byref(size), ctypes.c_uint64(ptr)) == 0
    assert base.value == ptr
    return size.value


@pytest.mark.parametrize("K", [128, 5120, 17408, 32768])
def test_pre_pass_stays_inside_the_scratch(pkg, synth, K):
    N = 272
    w = pkg.weights_from_numpy(*synth.make_weights(N, K, seed=K))
    s = pkg.gemv_scratch_alloc(K, N, 128, 16)
    size = _allocation_bytes(s.xf)
    # the same scratch with its first buffer inside a larger one, the rest of which nothing may touch
    buf = torch.full((size + GUARD,), 0x5A, dtype=torch.uint8, device="cuda")
    assert buf.data_ptr() % 256 == 0
    guarded = pkg.Scratch.from_buffer_copy(s)
    guarded.xf = buf.data_ptr()
    x = torch.randn((16, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(K)).to(torch.bfloat16)
    torch.cuda.synchronize()
    want = torch.empty((16, N), dtype=torch.bfloat16, device="cuda")
    for m in range(16):
        pkg.gemv_w4a16(want[m], w, x[m], s)
    for M in range(2, 17):
        y = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
        pkg.gemm_small_w4a16(y, w, x[:M], M, guarded)
        assert torch.equal(y.view(torch.int16), want[:M].view(torch.int16)), f"M = {M}"
        assert bool((buf[size:] == 0x5A).all()), f"M = {M} wrote behind the scratch"
    assert pkg.device_status() == 0
    pkg.gemv_scratch_free(s)
    pkg.awq_free(w)
