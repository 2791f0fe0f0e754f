"""The fused RMSNorm at M = 1 (inside the decode kernel) against the pre-pass of M >= 2: the row's sum of squares is added up in
one order everywhere, so a token's normalised activations and its outputs have the same bits alone and in a block."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from gpu_util import host_bits  # noqa: E402

pytestmark = pytest.mark.gpu


# one group; fewer units than groups per CTA; all groups in one batch of loads; more than one batch (over 52 groups); all 256 groups
@pytest.mark.parametrize("N,K", [(128, 128), (144, 896), (5120, 5120), (1040, 7168), (4096, 17408), (256, 32768)])
def test_normalised_row_alone_and_in_a_block(pkg, oracle, synth, N, K):
    packed, scale, zp = synth.make_weights(N, K, seed=N + K)
    w = pkg.weights_from_numpy(packed, scale, zp)
    scratch = pkg.gemv_scratch_alloc(K, N, 128, 16)
    gen = torch.Generator(device="cuda").manual_seed(K)
    x = torch.randn((3, K), device="cuda", generator=gen)
    x[:, :: max(1, K // 5)] *= 50.0
    x = x.to(torch.bfloat16)
    ln = (torch.randn(K, device="cuda", generator=gen) * 0.1).to(torch.bfloat16)
    torch.cuda.synchronize()
    y3 = torch.empty((3, N), dtype=torch.bfloat16, device="cuda")
    xn3 = torch.empty((3, K), dtype=torch.bfloat16, device="cuda")
    pkg.linear_fused(y3, w, x, 3, scratch, ln_weight=ln, xn_out=xn3)
    for m in range(3):
        y = torch.empty((1, N), dtype=torch.bfloat16, device="cuda")
        xn = torch.zeros((1, K), dtype=torch.bfloat16, device="cuda")
        plain = torch.empty(N, dtype=torch.bfloat16, device="cuda")
        pkg.linear_fused(y, w, x[m], 1, scratch, ln_weight=ln, xn_out=xn)
        pkg.gemv_w4a16(plain, w, xn[0], scratch)
        assert torch.equal(xn.view(torch.int16)[0], xn3.view(torch.int16)[m])
        assert torch.equal(y.view(torch.int16)[0], y3.view(torch.int16)[m])
        assert torch.equal(y.view(torch.int16)[0], plain.view(torch.int16))
    # against the formula in 64 bits: one rounding to bf16 apart where the fp32 sum of squares lands on the other side of a tie
    xd = x.double()
    want = (xd * torch.rsqrt((xd * xd).mean(dim=1, keepdim=True) + 1e-6) * (1.0 + ln.double())).to(torch.bfloat16)
    diff = (xn3.view(torch.int16).int() - want.view(torch.int16).int()).abs()
    assert int(diff.max()) <= 1 and float((diff != 0).float().mean()) < 0.01
    assert np.isfinite(host_bits(y3).astype(np.float32)).all() and pkg.device_status() == 0
    pkg.gemv_scratch_free(scratch)
    pkg.awq_free(w)


@pytest.mark.parametrize("M", [1, 2])
def test_normalised_call_that_adds_to_its_own_input(pkg, synth, M):
    """h += W norm(h) in place, at M = 1 too: the row is read before any of it is written."""
    N = K = 5120
    packed, scale, zp = synth.make_weights(N, K, seed=5)
    w = pkg.weights_from_numpy(packed, scale, zp)
    scratch = pkg.gemv_scratch_alloc(K, N, 128, 16)
    gen = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn((M, K), device="cuda", generator=gen).to(torch.bfloat16)
    ln = (torch.randn(K, device="cuda", generator=gen) * 0.1).to(torch.bfloat16)
    torch.cuda.synchronize()
    apart, own = x.clone(), x.clone()
    pkg.linear_fused(apart, w, x, M, scratch, ln_weight=ln, epilogue=pkg.EPILOGUE_RESIDUAL)
    pkg.linear_fused(own, w, own, M, scratch, ln_weight=ln, epilogue=pkg.EPILOGUE_RESIDUAL)
    assert torch.equal(apart.view(torch.int16), own.view(torch.int16)) and not torch.equal(own, x)
    assert pkg.device_status() == 0
    pkg.gemv_scratch_free(scratch)
    pkg.awq_free(w)
