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
def test_k_groups_and_splits(K, M):
    _check(512, K, M)


@pytest.mark.parametrize("N,K,M", [(5120, 1024, 777), (19072, 256, 520), (4736, 512, 2100)])
def test_several_tiles_per_cluster(N, K, M):
    _check(N, K, M)


@pytest.mark.parametrize("skew", [1, 4])
def test_output_not_16_byte_aligned(skew):
    _check(400, 384, 77, skew=skew)
    _check(2048, 1024, 300, skew=skew)
