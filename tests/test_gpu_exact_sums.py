"""The decode kernel's integer products, exactly: whole activations and scales of one make every output a whole number
below 2^24, which fp32 holds and bf16 rounds once, whatever the order of the sums. So each nibble (and int8 code) has to reach
the tensor core unchanged, at its own k, in its own row, and meet its own zero point. Every k group holds magnitudes from
1 to 2^11 or more, so that all three base-256 digits of an activation carry weight, and their sums have to meet the right powers."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# one group; a ragged last row tile; odd numbers of groups; segments of one group; more groups per CTA than ring stages
SHAPES = [(16, 128), (128, 128), (272, 384), (1040, 640), (19200, 256), (4096, 2176)]
MS = [1, 2, 5, 9, 12, 15, 16]


def _bf16(v):
    return torch.from_numpy(v.astype(np.float32)).cuda().to(torch.bfloat16)


def _activations(rng, K, big, rest, mids, step):
    """16 tokens; per group one large power of two (`big` in one group of each token), `mids` values of eight bits, small ones."""
    G = K // 128
    x = rng.integers(-8, 9, (16, K))
    for m in range(16):
        for g in range(G):
            at = 128 * g + rng.permutation(128)[:1 + mids]
            x[m, at[0]] = (big if g == m % G else rest) * rng.choice((-1, 1))
            x[m, at[1:]] = step * rng.integers(129, 256, mids) * rng.choice((-1, 1), mids)
        # the digits of the group with the large value: X = x 2^p with its largest magnitude at 2^21
        X = x[m].reshape(G, 128)[m % G] * (2 ** 21 // big)
        d0 = (X + 128) % 256 - 128
        d1 = ((X - d0) // 256 + 128) % 256 - 128
        d2 = (X - d0 - 256 * d1) // 65536
        assert all(np.count_nonzero(d) for d in (d0, d1, d2)) and len(np.unique(d0)) > 2 and len(np.unique(d1)) > 2
    return x


@pytest.mark.parametrize("N,K", SHAPES)
def test_int4_whole_numbers(pkg, synth, N, K):
    rng = np.random.Generator(np.random.PCG64(N + K))
    G = K // 128
    q = rng.integers(0, 16, (N, K), dtype=np.uint8)
    z = rng.integers(0, 16, (N, G), dtype=np.uint8)
    one = synth.f32_to_bf16_bits(np.ones((N, G), np.float32))
    w = pkg.weights_from_numpy(synth.pack_weight(q), one, synth.pack_zero_point(z))
    scratch = pkg.gemv_scratch_alloc(K, N, 128, 16)
    x = _activations(rng, K, 2 ** 18, 2 ** 14, 4, 8)
    v = (q.astype(np.int64) - np.repeat(z, 128, axis=1).astype(np.int64)).T
    want = x.astype(np.int64) @ v
    assert (np.abs(x).astype(np.int64) @ np.abs(v)).max() < 2 ** 24  # and so is every partial sum
    xd = _bf16(x)
    torch.cuda.synchronize()
    y32 = torch.empty(N, dtype=torch.float32, device="cuda")
    pkg.gemv_w4a16_f32(y32, w, xd[3], scratch)
    assert np.array_equal(y32.cpu().numpy().astype(np.int64), want[3])
    for M in MS:
        y = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
        pkg.gemm_small_w4a16(y, w, xd[:M], M, scratch)
        assert torch.equal(y, _bf16(want[:M])), f"M = {M}"
    assert pkg.device_status() == 0
    pkg.gemv_scratch_free(scratch)
    pkg.awq_free(w)


@pytest.mark.parametrize("N,K", SHAPES)
def test_int8_whole_numbers(pkg, N, K):
    rng = np.random.Generator(np.random.PCG64(N + K + 1))
    q = rng.integers(-127, 128, (N, K))
    q[:, ::128] = np.where(rng.integers(0, 2, (N, K // 128)) > 0, 127, -127)  # every group's largest: a scale of exactly one
    w = pkg.quantize_w8a16(_bf16(q))
    scratch = pkg.gemv_scratch_alloc(K, N, 128, 16)
    x = _activations(rng, K, 2 ** 15, 2 ** 11, 2, 2)
    want = x.astype(np.int64) @ q.astype(np.int64).T
    assert (np.abs(x).astype(np.int64) @ np.abs(q.astype(np.int64)).T).max() < 2 ** 24  # and so is every partial sum
    xd = _bf16(x)
    torch.cuda.synchronize()
    for M in MS:
        y = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
        if M == 1:
            pkg.gemv_w8a16(y, w, xd[0], scratch)
        else:
            pkg.gemm_small_w8a16(y, w, xd[:M], M, scratch)
        assert torch.equal(y, _bf16(want[:M])), f"M = {M}"
    assert pkg.device_status() == 0
    pkg.gemv_scratch_free(scratch)
    pkg.w8a16_free(w)
