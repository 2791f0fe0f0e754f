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
    the dequantised rows, weights within +-1 of their zero points, activations that bring the sums back to ordinary size. (Every
    scale is of one size here; the next test mixes them within a warp and looks at every weight by itself.)"""
    N, K, M = 144, 640, 40
    rng = np.random.Generator(np.random.PCG64(5))
    z = rng.integers(1, 15, (N, K // 128), dtype=np.uint8)
    q = (np.repeat(z, 128, axis=1).astype(np.int64) + rng.integers(-1, 2, (N, K))).astype(np.uint8)
    scale = synth.f32_to_bf16_bits(np.full((N, K // 128), np.ldexp(1.5, exponent), np.float32))
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


# bf16 bits: subnormal, the smallest normal, ordinary, the last one below 2^126, from 2^126 up to the largest; either sign; zeros
SCALES = [0x0000, 0x8000, 0x0001, 0x0055, 0x007F, 0x0080, 0x00C1, 0x3C23, 0x3E80, 0x5F35, 0x7D80, 0x7DFF, 0x7E00, 0x7E7F, 0x7E80,
          0x7E81, 0x7EFF, 0x7F00, 0x7F40, 0x7F7F]
SCALES += [s | 0x8000 for s in SCALES[2:]]


def _one_weight_per_output(N, K, seed):
    """Codes, zero points and scale bits; every weight finite. Scales are drawn per (row, group), so that a warp's 32 rows mix them."""
    rng = np.random.Generator(np.random.PCG64(seed))
    G = K // 128
    scale = rng.choice(np.array(SCALES, np.uint16), (N, G))
    z = rng.integers(0, 16, (N, G), dtype=np.uint8)
    s = np.abs(synth.bf16_bits_to_f32(scale).astype(np.float64))
    reach = np.repeat(np.minimum(15, np.floor(2.0 ** 128 * (1 - 2.0 ** -9) / np.maximum(s, 2.0 ** -140))).astype(np.int64), 128, axis=1)
    zk = np.repeat(z.astype(np.int64), 128, axis=1)
    q = np.clip(rng.integers(0, 16, (N, K)), zk - reach, zk + reach).astype(np.uint8)
    return q, z, scale


# narrow tiles in one piece and in four; 128 tokens in four; 224 and 256, whose weight rings have four stages
@pytest.mark.parametrize("N,K,M,splits,tokens", [(144, 256, 128, 1, 32), (272, 4096, 224, 4, 32), (2192, 4096, 128, 4, 128),
                                                 (9488, 1024, 224, 1, 224), (9488, 512, 256, 1, 256)])
def test_every_weight_by_itself(N, K, M, splits, tokens):
    """Activations with one power of two per token: an output is one weight times it, exactly, whatever the order of the sum. So the
    weights inside the kernel are compared value for value with bf16((q - zp) s), for every (q, zp) and scales of every kind. Two
    powers, so that every weight but zero lands in bf16's normal range under one of them."""
    assert pkg.prefill_plan(M, N, K) == (tokens, splits)
    q, z, scale = _one_weight_per_output(N, K, seed=N + K)
    zk, sk = np.repeat(z.astype(np.int64), 128, axis=1), np.repeat(scale, 128, axis=1)
    ordinary = (sk & 0x7FFF) < 0x7E00
    assert np.unique(q[ordinary].astype(np.int64) * 16 + zk[ordinary]).size == 256
    exact = (q.astype(np.int64) - zk) * synth.bf16_bits_to_f32(sk).astype(np.float64)  # twelve bits at the most: exact in fp32, too
    bits = synth.f32_to_bf16_bits(exact.astype(np.float32))
    assert ((bits & 0x7FFF) < 0x7F80).all()
    w = pkg.weights_from_numpy(synth.pack_weight(q), scale, synth.pack_zero_point(z))
    deq = torch.empty((N, K), dtype=torch.bfloat16, device="cuda")
    pkg.w4a16_dequant_rows(deq, w, 0, N)
    want = torch.from_numpy(bits.view(np.int16)).cuda().view(torch.bfloat16)
    nonzero = want != 0
    assert torch.equal(deq == 0, ~nonzero) and torch.equal(deq[nonzero].view(torch.int16), want[nonzero].view(torch.int16))
    ws = pkg.gemm_workspace_alloc(4096)
    seen = torch.zeros((N, K), dtype=torch.bool, device="cuda")
    for power in (2.0 ** 60, 2.0 ** -60):
        for k0 in range(0, K, M):
            n = min(M, K - k0)
            x = torch.zeros((M, K), dtype=torch.bfloat16, device="cuda")
            x[torch.arange(n), torch.arange(k0, k0 + n)] = power
            c = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
            pkg.gemm_w4a16(c, w, x, M, ws)
            got, ref = c[:n].double().t(), want[:, k0:k0 + n].double() * power
            normal = (ref.abs() >= 2.0 ** -126) & (ref.abs() < 2.0 ** 128)
            assert torch.equal(got[normal], ref[normal])
            assert bool((got[ref == 0] == 0).all())
            seen[:, k0:k0 + n] |= normal
    assert torch.equal(seen, nonzero) and pkg.device_status() == 0
    pkg.gemm_workspace_free(ws)
    pkg.awq_free(w)


def test_scales_that_are_no_numbers():
    """An infinite scale makes weights infinite, a NaN its row; rows beside them, in the same warp, keep their sums."""
    N, K, M = 144, 256, 40
    rng = np.random.Generator(np.random.PCG64(6))
    z = rng.integers(0, 8, (N, K // 128), dtype=np.uint8)
    q = (np.repeat(z, 128, axis=1).astype(np.int64) + rng.integers(1, 8, (N, K))).astype(np.uint8)  # no weight is zero
    scale = np.full((N, K // 128), 0x3F80, np.uint16)
    for row, bits in ((3, 0x7F80), (40, 0xFF80), (75, 0x7FC0), (130, 0x7F80)):
        scale[row, 1] = bits
    scale[5, 1] = scale[41, 1] = 0x7F00  # a large one beside them
    q[[5, 41]] = np.repeat(z, 128, axis=1)[[5, 41]] + 1
    w = pkg.weights_from_numpy(synth.pack_weight(q), scale, synth.pack_zero_point(z))
    # no activation is zero, as zero times an infinite weight is NaN
    x = torch.full((M, K), 2.0 ** -7, dtype=torch.bfloat16, device="cuda")
    x[:, :128] = 2.0 ** -8
    ws = pkg.gemm_workspace_alloc(4096)
    c = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    pkg.gemm_w4a16(c, w, x, M, ws)
    v = (q.astype(np.int64) - np.repeat(z, 128, axis=1)).astype(np.float64) * np.repeat(synth.bf16_bits_to_f32(scale), 128, axis=1)
    with np.errstate(invalid="ignore"):
        ref = torch.from_numpy(v @ x[0].double().cpu().numpy()).to(torch.float32).to(torch.bfloat16).cuda()
    assert bool(torch.isposinf(c[:, [3, 130]]).all()) and bool(torch.isneginf(c[:, 40]).all()) and bool(torch.isnan(c[:, 75]).all())
    rest = torch.isfinite(ref)
    assert int(rest.sum()) == N - 4
    # sums of whole numbers over 2^8, below 2^4: exact; and 128 equal terms of 2^120 with small ones that vanish in every order
    assert torch.equal(c[:, rest], ref[rest].expand(M, -1))
    assert pkg.device_status() == 0
    pkg.gemm_workspace_free(ws)
    pkg.awq_free(w)
