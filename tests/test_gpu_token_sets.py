"""Every token-set split of the decode kernel (M = 2..16) against its M = 1 form: the same unit ranges, the same order
of the same fp32 operations per token, so every row has to come out bit for bit as the row alone does."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _run(pkg, w, x, scratch):
    M, N = x.shape[0], w.out_f
    y = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    pkg.gemm_small_w4a16(y, w, x, M, scratch)
    return y


# one k group; an odd number of groups; split tiles with a ragged last row tile; more tiles than CTAs
@pytest.mark.parametrize("N,K", [(16, 128), (144, 896), (1040, 2176), (19200, 640)])
def test_rows_equal_the_single_row_kernel(pkg, synth, N, K):
    packed, scale, zp = synth.make_weights(N, K, seed=N + K)
    w = pkg.weights_from_numpy(packed, scale, zp)
    scratch = pkg.gemv_scratch_alloc(K, N, 128, 16)
    gen = torch.Generator(device="cuda").manual_seed(K)
    x = torch.randn((16, K), device="cuda", generator=gen)
    x[:, :: max(1, K // 7)] *= 300.0
    x = x.to(torch.bfloat16)
    torch.cuda.synchronize()
    rows = torch.empty((16, N), dtype=torch.bfloat16, device="cuda")
    for m in range(16):
        pkg.gemv_w4a16(rows[m], w, x[m], scratch)
    for M in range(2, 17):
        y = _run(pkg, w, x[:M], scratch)
        assert torch.equal(y.view(torch.int16), rows[:M].view(torch.int16)), f"M = {M}"
    assert pkg.device_status() == 0
    pkg.gemv_scratch_free(scratch)
    pkg.awq_free(w)


# int8 weights: tiles of two to about twenty pieces, whose reader differs by token count; twice, so that the second launch finds
# the words that the first one has zeroed
@pytest.mark.parametrize("N,K", [(272, 4096), (1024, 16384), (5120, 640)])
@pytest.mark.parametrize("M", [2, 3, 4, 8, 12, 13, 14, 15, 16])
def test_int8_rows_of_split_tiles(pkg, N, K, M):
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    w = pkg.quantize_w8a16((torch.randn((N, K), device="cuda", generator=gen) * 0.02).to(torch.bfloat16))
    scratch = pkg.gemv_scratch_alloc(K, N, 128, 16)
    x = torch.randn((M, K), device="cuda", generator=gen).to(torch.bfloat16)
    rows, y = (torch.empty((M, N), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    for m in range(M):
        pkg.gemv_w8a16(rows[m], w, x[m], scratch)
    for _ in range(2):
        y.zero_()
        pkg.gemm_small_w8a16(y, w, x, M, scratch)
        assert torch.equal(y.view(torch.int16), rows.view(torch.int16))
    assert pkg.device_status() == 0
    pkg.gemv_scratch_free(scratch)
    pkg.w8a16_free(w)
