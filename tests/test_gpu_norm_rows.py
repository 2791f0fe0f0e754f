"""The fused RMSNorm at M = 1 (inside the decode kernel) and in the pre-pass of M >= 2: the row's sum of squares is added up in
one order everywhere, 32 chains over the k groups and then a tree, so a token's normalised activations and its outputs have the
same bits alone and in a block, and the bits of that order."""
import pytest

torch = pytest.importorskip("torch")
from gpu_util import captured_edges  # noqa: E402

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
    assert bool(torch.isfinite(y3.float()).all()) and pkg.device_status() == 0
    pkg.gemv_scratch_free(scratch)
    pkg.awq_free(w)


def _chains(x):
    """Sum of squares per row: chain l takes elements 4 l .. 4 l + 3 of every group, groups ascending; then the xor tree."""
    q = (x.float() ** 2).view(x.shape[0], -1, 32, 4)
    v = (q[..., 0] + q[..., 1]) + (q[..., 2] + q[..., 3])
    ss = torch.zeros_like(v[:, 0])
    for g in range(v.shape[1]):
        ss = ss + v[:, g]
    lanes = torch.arange(32, device=x.device)
    for off in (16, 8, 4, 2, 1):
        ss = ss + ss[:, lanes ^ off]
    return ss[:, :1]


def _by_groups(x):
    return (x.float() ** 2).view(x.shape[0], -1, 128).sum(dim=2).sum(dim=1, keepdim=True)


# one group; groups that fill the chains' rounds of loads and that do not; all 256 groups
@pytest.mark.parametrize("K", [128, 640, 5120, 7040, 17408, 32768])
@pytest.mark.parametrize("M", [1, 3, 16])
def test_order_of_the_sum_of_squares(pkg, synth, M, K):
    N, eps = 256, 1e-6
    w = pkg.weights_from_numpy(*synth.make_weights(N, K, seed=3))
    scratch = pkg.gemv_scratch_alloc(K, N, 128, 16)
    gen = torch.Generator(device="cuda").manual_seed(K + M)
    ln = torch.randn(K, device="cuda", generator=gen).to(torch.bfloat16)
    smooth = torch.randn((M, K), device="cuda", generator=gen).to(torch.bfloat16)
    # every chain reaches 2^24 in the first group, and the ones that follow are lost one by one (a sum of several is not)
    steep = torch.full((M, K), 0.5, device="cuda", dtype=torch.bfloat16)
    steep[:, :128] = 0.0
    steep[:, :128:4] = 4096.0
    n, e = torch.tensor(float(K), device="cuda"), torch.tensor(eps, device="cuda", dtype=torch.float32)

    def norm(x, ss):
        return (x.float() * torch.rsqrt(ss / n + e) * (1.0 + ln.float())).to(torch.bfloat16).view(torch.int16)

    for x in (smooth, steep):
        y = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
        xn = torch.zeros((M, K), dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        pkg.linear_fused(y, w, x, M, scratch, ln_weight=ln, ln_eps=eps, xn_out=xn)
        assert torch.equal(xn.view(torch.int16), norm(x, _chains(x)))
    if K >= 17408:  # where the order shows in bf16
        assert not torch.equal(norm(steep, _chains(steep)), norm(steep, _by_groups(steep)))
    assert pkg.device_status() == 0
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


@pytest.mark.parametrize("max_m", [1, 16])
@pytest.mark.parametrize("H", [128, 1152, 5120])
def test_plain_calls_whose_output_overlaps_the_input(pkg, synth, H, max_m):
    """The same for calls without a norm at M = 1, whatever the scratch has room for: a pre-pass kernel reads x first."""
    w = pkg.weights_from_numpy(*synth.make_weights(H, H, seed=6))
    scratch = pkg.gemv_scratch_alloc(H, H, 128, max_m)
    gen = torch.Generator(device="cuda").manual_seed(H)
    x = torch.randn(H, device="cuda", generator=gen).to(torch.bfloat16)
    plain, res, wide = torch.empty_like(x), x.clone(), torch.empty(H, device="cuda")
    torch.cuda.synchronize()
    pkg.gemv_w4a16(plain, w, x, scratch)
    pkg.gemv_w4a16_f32(wide, w, x, scratch)
    pkg.linear_fused(res, w, x, 1, scratch, epilogue=pkg.EPILOGUE_RESIDUAL)
    own = torch.zeros(2 * H, device="cuda", dtype=torch.bfloat16)  # x lies in the second half, which a y of 32 bits reaches
    xo = own[H:]

    def gemv(st):
        pkg.gemv_w4a16(xo, w, xo, scratch, stream=st)

    def gemv_static(st):
        pkg.gemv_w4a16_static(xo, w, xo, stream=st)

    def gemv_f32(st):
        pkg.gemv_w4a16_f32(own.view(torch.float32), w, xo, scratch, stream=st)

    def residual(st):
        pkg.linear_fused(xo, w, xo, 1, scratch, epilogue=pkg.EPILOGUE_RESIDUAL, stream=st)

    for call, got, want in ((gemv, xo, plain), (gemv_static, xo, plain), (gemv_f32, own.view(torch.float32), wide), (residual, xo, res)):
        xo.copy_(x)
        call(torch.cuda.current_stream())
        assert torch.equal(got.view(torch.int16), want.view(torch.int16)), call.__name__
        assert len(captured_edges(call)) == 1  # two kernels
    assert len(captured_edges(lambda st: pkg.gemv_w4a16(plain, w, x, scratch, stream=st))) == 0
    pkg.gemv_w4a16(plain, w, x, scratch)  # the scratch serves an ordinary call as before
    xo.copy_(x)
    gemv(torch.cuda.current_stream())
    assert torch.equal(xo, plain) and pkg.device_status() == 0
    pkg.gemv_scratch_free(scratch)
    pkg.awq_free(w)


@pytest.mark.parametrize("M", [1, 3])
def test_normalised_rows_must_not_go_over_the_input(pkg, synth, M):
    H = 1024
    w = pkg.weights_from_numpy(*synth.make_weights(H, H, seed=7))
    scratch = pkg.gemv_scratch_alloc(H, H, 128, 16)
    buf = torch.randn(3 * M * H, device="cuda").to(torch.bfloat16)
    x, ln, y = buf[M * H:2 * M * H], torch.zeros(H, device="cuda", dtype=torch.bfloat16), torch.empty((M, H), device="cuda", dtype=torch.bfloat16)
    before = buf.clone()
    for at in (M * H, 8, 2 * M * H - 8):  # x itself, and one step of 16 bytes into either end
        with pytest.raises(pkg.W4A16Error, match="overlaps"):
            pkg.linear_fused(y, w, x, M, scratch, ln_weight=ln, xn_out=buf[at:at + M * H])
    assert torch.equal(buf, before)
    pkg.linear_fused(y, w, x, M, scratch, xn_out=x)  # without the norm nothing is stored there
    for at in (0, 2 * M * H):  # right in front of x and right behind it
        xn = buf[at:at + M * H]
        pkg.linear_fused(y, w, x, M, scratch, ln_weight=ln, xn_out=xn)
        assert torch.equal(x, before[M * H:2 * M * H]) and not torch.equal(xn, before[at:at + M * H])
    assert pkg.device_status() == 0
    pkg.gemv_scratch_free(scratch)
    pkg.awq_free(w)
