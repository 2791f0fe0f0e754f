"""The load path (checkpoint tensors -> stream -> bf16 rows) at the edges of its kernels' tiles: row blocks of 128 and
16, blocks of eight k groups, row offsets that straddle row tiles, every bf16 scale. Whole values: bit-exact."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _tensors(rows, cols, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    lo, hi = -2 ** 31, 2 ** 31 - 1
    groups = cols // 128
    packed = torch.randint(lo, hi, (rows, cols // 8), dtype=torch.int32, device="cuda", generator=gen)
    scale = (torch.randn((rows, groups), device="cuda", generator=gen) * 0.02).to(torch.bfloat16)
    zp = torch.randint(lo, hi, (rows // 8, groups), dtype=torch.int32, device="cuda", generator=gen)
    return packed, scale, zp


def _expected(packed, scale, zp):
    """bf16((q - zp) * s), the product exact in fp32 and rounded once."""
    rows, cols = packed.shape[0], packed.shape[1] * 8
    sh = torch.arange(0, 32, 4, device="cuda", dtype=torch.int32)
    q = ((packed.unsqueeze(-1) >> sh) & 15).view(rows, cols)
    z = ((zp.unsqueeze(1) >> sh.view(1, 8, 1)) & 15).reshape(rows, -1)
    d = (q - z.repeat_interleave(128, 1)).float() * scale.float().repeat_interleave(128, 1)
    return d.to(torch.bfloat16)


def _same(a, b):
    return torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("rows", [16, 112, 128, 144, 272])
@pytest.mark.parametrize("cols", [128, 896, 1024, 1152])
def test_round_trip_edges(pkg, rows, cols):
    t = _tensors(rows, cols, rows + cols)
    want = _expected(*t)
    w = pkg.awq_repack(*t)
    for row0, n in [(0, rows), (0, 1), (rows - 1, 1), (5, min(18, rows - 5)), (3, rows - 3)]:
        out = torch.full((n + 1, cols), 7.0, dtype=torch.bfloat16, device="cuda")
        pkg.w4a16_dequant_rows(out, w, row0, n)
        assert _same(out[:n], want[row0:row0 + n]) and bool((out[n] == 7).all())
    pkg.awq_free(w)


def test_pieces_that_straddle_row_tiles(pkg):
    cols, parts = 1152, [16, 144, 80, 272]
    w = pkg.awq_alloc_fused(sum(parts), cols)
    want, at = [], 0
    for i, n in enumerate(parts):
        t = _tensors(n, cols, i)
        pkg.awq_repack_into(w, at, *t)
        want.append(_expected(*t))
        at += n
    out = torch.empty((at, cols), dtype=torch.bfloat16, device="cuda")
    pkg.w4a16_dequant_rows(out, w, 0, at)
    assert _same(out, torch.cat(want))
    pkg.awq_free(w)


def test_interleaved_gate_up(pkg):
    inter, cols = 144, 1152
    gate, up = _tensors(inter, cols, 1), _tensors(inter, cols, 2)
    w = pkg.awq_alloc_fused(2 * inter, cols)
    pkg.awq_repack_into_swiglu(w, 0, *gate, inter)
    pkg.awq_repack_into_swiglu(w, inter, *up, inter)
    out = torch.empty((2 * inter, cols), dtype=torch.bfloat16, device="cuda")
    pkg.w4a16_dequant_rows(out, w, 0, 2 * inter)
    assert _same(out[0::2], _expected(*gate)) and _same(out[1::2], _expected(*up))
    pkg.awq_free(w)


def test_every_scale(pkg):
    """All 65536 bf16 scales (subnormals, infinities and NaN among them; a NaN only has to stay one)."""
    rows, cols = 4096, 16 * 128
    packed, _, zp = _tensors(rows, cols, 3)
    scale = torch.from_numpy(np.arange(65536, dtype=np.uint16).view(np.int16)).cuda().view(torch.bfloat16).view(rows, 16)
    want = _expected(packed, scale, zp)
    w = pkg.awq_repack(packed, scale, zp)
    out = torch.empty((rows, cols), dtype=torch.bfloat16, device="cuda")
    pkg.w4a16_dequant_rows(out, w, 0, rows)
    nan = torch.isnan(want)
    assert torch.equal(nan, torch.isnan(out))
    assert _same(out.masked_fill(nan, 0), want.masked_fill(nan, 0))
    pkg.awq_free(w)
