"""Calls without a `stream` go to the stream that is current in the calling thread."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_calls_follow_the_current_stream(pkg, synth):
    packed, scale, zp = synth.make_weights(1040, 640, seed=3)
    w = pkg.weights_from_numpy(packed, scale, zp)
    scratch = pkg.gemv_scratch_alloc(640, 1040, 128, 16)
    x = torch.randn((9, 640), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).to(torch.bfloat16)
    want, got = torch.empty((9, 1040), dtype=torch.bfloat16, device="cuda"), torch.zeros((9, 1040), dtype=torch.bfloat16, device="cuda")
    pkg.gemm_small_w4a16(want, w, x, 9, scratch)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    assert pkg._stream() == torch.cuda.current_stream().cuda_stream
    with torch.cuda.stream(side):
        assert pkg._stream() == side.cuda_stream
        pkg.gemm_small_w4a16(got, w, x, 9, scratch)
    assert pkg._stream(side) == side.cuda_stream
    side.synchronize()
    assert torch.equal(got, want) and pkg.device_status() == 0
    pkg.gemv_scratch_free(scratch)
    pkg.awq_free(w)
