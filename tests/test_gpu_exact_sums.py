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


# ---- the digits' sums above 2^24, where fp32 no longer holds 256 D1 + D0: how the three are put together decides the last bits
def _digits(X):
    d0 = (X + 128) % 256 - 128
    d1 = ((X - d0) // 256 + 128) % 256 - 128
    return d0, d1, (X - d0 - 256 * d1) // 65536


def _f32(v):
    return v.astype(np.float32).astype(np.float64)


def _fixup(X, wt, z, join=lambda low: _f32(low)):
    """One k group, scale one: fp32(65536 D2 + fp32(256 D1 + D0)) - z fp32(sum of X), every step rounded once (products and sums of
    these sizes are exact in fp64). X [M, 128], wt [N, 128] as the tensor core has it, z [N]."""
    d0, d1, d2 = (d @ wt.T for d in _digits(X))
    dot = _f32(65536.0 * d2 + join(256 * d1 + d0))
    return _f32(dot - z * _f32(X.sum(1, keepdims=True))), np.abs(256 * d1 + d0)


def _cancelling(rng, N, base, powers, lo, hi, wmin, wmax):
    """X [16, 128] with about a hundred values near 2^15 (digits d1 of full size), base^0 .. base^(powers - 1) and 2^21, the group's
    largest (so X is x itself); row n's weights cancel token n % 16 down to a remainder below 128, so that an error in the
    last bits of the sums is all that is left. One place holds the largest weight and no activation (int8: a row's scale of one)."""
    X = np.zeros((16, 128), np.int64)
    W = np.zeros((N, 128), np.int64)
    at = rng.permutation(128)
    fix, top, idle, mid = at[:powers], at[powers], at[powers + 1], at[powers + 2:]
    X[:, fix], X[:, top] = base ** np.arange(powers), 2 ** 21
    for m in range(16):
        X[m, mid] = 2 ** 7 * rng.integers(200, 256, mid.size)  # eight significant bits each
        X[m, mid[:20]] = rng.integers(1, 256, 20)
    W[:, idle] = wmax
    for n in range(N):
        W[n, mid] = rng.integers(lo, hi, mid.size)
        rest = int(rng.integers(1, 128)) - int(X[n % 16, mid] @ W[n, mid])
        W[n, top] = round(rest / 2 ** 21)
        rest -= int(W[n, top]) * 2 ** 21
        for i in range(powers):
            W[n, fix[i]] = rest if i == powers - 1 else (rest + base // 2) % base - base // 2
            rest = (rest - int(W[n, fix[i]])) // base
    assert W.min() >= wmin and W.max() <= wmax
    return X, W


def _truncated(low):
    """What the device must not do: the joined sum cut to 24 bits instead of rounded."""
    s = np.maximum(np.floor(np.log2(np.maximum(np.abs(low), 1))) - 23, 0)
    return np.trunc(low / 2.0 ** s) * 2.0 ** s


def _check_last_bits(X, wt, z, call):
    want, low = _fixup(X, wt, z)
    own = np.arange(16)[:, None] == np.arange(wt.shape[0])[None, :] % 16
    assert low[own].min() > 2 ** 24
    cut = _fixup(X, wt, z, _truncated)[0]
    assert (_bf16(want) != _bf16(cut)).cpu().numpy()[own].mean() > 0.1  # these inputs tell the two apart
    xd = _bf16(X)
    torch.cuda.synchronize()
    for M in range(1, 17):
        y = torch.empty((M, wt.shape[0]), dtype=torch.bfloat16, device="cuda")
        call(y, xd[:M], M)
        assert torch.equal(y, _bf16(want[:M])), f"M = {M}"


def test_int4_sums_past_24_bits(pkg, synth):
    N = 272
    X, W = _cancelling(np.random.Generator(np.random.PCG64(24)), N, 16, 6, 4, 8, -8, 7)
    one, z = synth.f32_to_bf16_bits(np.ones((N, 1), np.float32)), np.full((N, 1), 8, np.uint8)
    q = W + 8
    w = pkg.weights_from_numpy(synth.pack_weight(q.astype(np.uint8)), one, synth.pack_zero_point(z))
    s = pkg.gemv_scratch_alloc(128, N, 128, 16)
    _check_last_bits(X, q, 8.0, lambda y, x, M: pkg.gemv_w4a16(y, w, x, s) if M == 1 else pkg.gemm_small_w4a16(y, w, x, M, s))
    assert pkg.device_status() == 0
    pkg.gemv_scratch_free(s)
    pkg.awq_free(w)


def test_int8_sums_past_24_bits(pkg):
    N = 272
    X, W = _cancelling(np.random.Generator(np.random.PCG64(25)), N, 128, 3, 40, 100, -127, 127)
    w = pkg.quantize_w8a16(_bf16(W))
    s = pkg.gemv_scratch_alloc(128, N, 128, 16)
    _check_last_bits(X, W, 0.0, lambda y, x, M: pkg.gemv_w8a16(y, w, x, s) if M == 1 else pkg.gemm_small_w8a16(y, w, x, M, s))
    assert pkg.device_status() == 0
    pkg.gemv_scratch_free(s)
    pkg.w8a16_free(w)
