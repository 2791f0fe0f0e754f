"""The prefill GEMM at the edges of its launch shapes: row tiles of 128 in pairs, token tiles of 32..256 with a
ragged last one, K split over a cluster, and outputs that do not take 16-byte stores."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

pkg = importlib.import_module("qwen38-3090-cuda-server_b200")
synth = importlib.import_module("qwen38-3090-cuda-server_b200.synth")


def _layer(N, K, seed):
    packed, scale, zp = synth.make_weights(N, K, seed=seed)
    w = pkg.weights_from_numpy(packed, scale, zp)
    deq = torch.empty((N, K), dtype=torch.bfloat16, device="cuda")
    pkg.w4a16_dequant_rows(deq, w, 0, N)
    return w, deq


def _check(N, K, M, skew=0):
    """The product against fp64 on the same bf16 weights. Each output is one rounding to bf16 (2^-9 relative) of an
    fp32 sum of K products, so an element may be off by 2^-8 of its value (a rounding and its neighbour) plus the fp32
    sum's error, K * 2^-24 of the sum of magnitudes at the most."""
    w, deq = _layer(N, K, seed=N + K + M)
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn((M, K), device="cuda", generator=gen).to(torch.bfloat16)
    ws = pkg.gemm_workspace_alloc(4096)
    buf = torch.full((skew + M * N + 64,), 7.0, dtype=torch.bfloat16, device="cuda")
    c = buf[skew:skew + M * N].view(M, N)
    pkg.gemm_w4a16(c, w, x, M, ws)
    first = c.clone()
    pkg.gemm_w4a16(c, w, x, M, ws)
    assert pkg.device_status() == 0
    assert torch.equal(first, c), "two runs differ"
    assert bool((buf[:skew] == 7).all()) and bool((buf[skew + M * N:] == 7).all()), "wrote outside C"
    ref = x.double() @ deq.double().t()
    mag = x.double().abs() @ deq.double().abs().t()
    assert bool(((c.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + K * 2.0 ** -24 * mag).all())
    pkg.gemm_workspace_free(ws)
    pkg.awq_free(w)


@pytest.mark.parametrize("N", [16, 128, 144, 256, 272, 400])
@pytest.mark.parametrize("M", [1, 31, 33, 256, 257])
def test_row_and_token_edges(N, M):
    _check(N, 384, M)


@pytest.mark.parametrize("K", [128, 256, 640, 2176])
@pytest.mark.parametrize("M", [17, 96, 193, 300])
def test_k_groups_in_one_piece(K, M):
    assert pkg.prefill_plan(M, 512, K)[1] == 1
    _check(512, K, M)


# Layers of few tiles and many k groups, which take 2, 3 or 4 splits: odd numbers of row tiles and a last one of 16 rows,
# ragged token tiles, several of them, k groups that do not divide, outputs that do not take 16-byte stores.
SPLIT = [(16, 4096, 33, 0), (272, 4096, 1, 0), (272, 5120, 300, 1), (400, 17408, 77, 0), (1040, 4224, 130, 4),
         (5120, 4096, 77, 0), (5120, 17408, 17, 0), (5120, 17408, 200, 1), (8192, 4224, 77, 0), (8192, 5120, 100, 0)]


@pytest.mark.parametrize("N,K,M,skew", SPLIT)
def test_split_k(N, K, M, skew):
    assert pkg.prefill_plan(M, N, K)[1] > 1
    _check(N, K, M, skew)


def test_split_cases_cover_every_count():
    assert {pkg.prefill_plan(M, N, K)[1] for N, K, M, _ in SPLIT} == {2, 3, 4}


def test_the_plan_is_fixed():
    """The number of splits decides a row's bits, so it must not follow the device: 33, 22 and 15 clusters of four, six
    and eight CTAs are what the plan goes by (the first two shapes are one row pair beyond 33 clusters and just within)."""
    want = [(64, 8704, 5120, 32, 1), (64, 8448, 5120, 64, 2), (300, 2048, 4096, 96, 2), (130, 1040, 4224, 64, 4),
            (77, 5120, 17408, 96, 3), (777, 5120, 8192, 128, 1), (4096, 34816, 5120, 256, 1)]
    assert [pkg.prefill_plan(M, N, K) for M, N, K, _, _ in want] == [w[3:] for w in want]


@pytest.mark.parametrize("K", [512, 4096])
def test_a_row_depends_on_the_splits_only(K):
    """Calls with the same number of splits give a row the same bits, whatever M and the tile."""
    N = 400
    w, _ = _layer(N, K, seed=7)
    x = torch.randn((1300, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(7)).to(torch.bfloat16)
    ws = pkg.gemm_workspace_alloc(4096)
    first, tokens = {}, {}
    for M in (1, 33, 77, 130, 300, 520, 1000, 1300):
        tn, splits = pkg.prefill_plan(M, N, K)
        c = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
        pkg.gemm_w4a16(c, w, x[:M], M, ws)
        seen = first.setdefault(splits, c)
        tokens.setdefault(splits, set()).add(tn)
        n = min(M, seen.shape[0])
        assert torch.equal(c[:n].view(torch.int16), seen[:n].view(torch.int16)), (M, tn, splits)
        if M > seen.shape[0]:
            first[splits] = c
    assert pkg.device_status() == 0 and any(len(t) > 1 for t in tokens.values())
    pkg.gemm_workspace_free(ws)
    pkg.awq_free(w)


@pytest.mark.parametrize("N,K,M", [(5120, 1024, 777), (19072, 256, 520), (4736, 512, 2100)])
def test_several_tiles_per_cluster(N, K, M):
    _check(N, K, M)


@pytest.mark.parametrize("skew", [1, 4])
def test_output_not_16_byte_aligned(skew):
    _check(400, 384, 77, skew=skew)
    _check(2048, 1024, 300, skew=skew)


@pytest.mark.parametrize("exponent", [-126, -20, 125, 126, 127])
def test_scales_at_both_ends(exponent):
    """The product with scales up to the largest powers of two (from 2^126 on four times the scale is no number) against fp64 on
    the dequantised rows, weights within +-1 of their zero points, activations that bring the sums back to ordinary size."""
    N, K, M = 144, 640, 40
    rng = np.random.Generator(np.random.PCG64(5))
    z = rng.integers(1, 15, (N, K // 128), dtype=np.uint8)
    q = (np.repeat(z, 128, axis=1).astype(np.int64) + rng.integers(-1, 2, (N, K))).astype(np.uint8)
    scale = synth.f32_to_bf16_bits(np.full((N, K // 128), np.ldexp(1.5, exponent), np.float32))
    scale[::3, 1] = synth.f32_to_bf16_bits(np.array([0.25], np.float32))[0]  # rows of both kinds in a warp
    w = pkg.weights_from_numpy(synth.pack_weight(q), scale, synth.pack_zero_point(z))
    deq = torch.empty((N, K), dtype=torch.bfloat16, device="cuda")
    pkg.w4a16_dequant_rows(deq, w, 0, N)
    x = torch.randn((M, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    x = (x * 2.0 ** (-60 if exponent > 0 else 20)).to(torch.bfloat16)
    ws = pkg.gemm_workspace_alloc(4096)
    c = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    pkg.gemm_w4a16(c, w, x, M, ws)
    ref, mag = x.double() @ deq.double().t(), x.double().abs() @ deq.double().abs().t()
    assert pkg.device_status() == 0 and bool(torch.isfinite(c).all())
    assert bool(((c.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + K * 2.0 ** -24 * mag).all())
    pkg.gemm_workspace_free(ws)
    pkg.awq_free(w)
