"""Index tables of at most 16 entries counted instead of gathered, and the wide cast-and-transpose tiles."""

import pytest
import torch

import cases as C
from oracle import quantizers as OQ
from oracle import tables as OT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [2, 3, 9, 16])
@pytest.mark.parametrize("shape,block", [((1, 8), 8), ((3, 192), 64), ((1000, 320), 64), ((640, 2048), 16)])
@pytest.mark.parametrize("pot", [False, True])
def test_quantize_mx_to_indices(levels, shape, block, pot):
    import voyager_b200 as vb

    g = torch.Generator().manual_seed(levels + shape[1])
    grid = torch.sort(torch.randn(levels, generator=g) * 10).values.bfloat16()
    values = torch.arange(1 << 16, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    mid = ((grid[:-1].float() + grid[1:].float()) / 2)
    index = torch.searchsorted(mid, values.float()).to(torch.int64)
    x = C.randn(shape[0], *shape, outliers=0.002)
    x.view(-1)[:: 97] *= 2.0 ** -120
    x[0, :8] = 0.0
    if shape[0] > 2:
        x[1, 3], x[2, 5] = float("inf"), float("nan")
    spec = vb.rounding.table_round(index.cuda())
    assert spec.mode == vb._native.ROUND_TABLE and spec.c.n_edges == levels - 1
    scale_table = None if pot else OT.quantization_map("fp8_e5m3")
    want_s, want_c = OQ.quantize_mx(x, index, [-1], block, 31.0, pot, scale_table, mid)
    got_s, got_c = torch.ops.quantized_ops.quantize_mx(x.cuda(), index.cuda(), [-1], block, 31.0, pot,
                                                       None if pot else scale_table.cuda(), mid.cuda())
    assert torch.equal(got_s.cpu().view(torch.int16), want_s.view(torch.int16))
    assert torch.equal(got_c.cpu().view(torch.int16), want_c.view(torch.int16))


@pytest.mark.parametrize("rows,cols", [(1, 8), (16, 128), (127, 136), (130, 264), (128, 1000), (388, 512), (333, 40)])
@pytest.mark.parametrize("fmt", ["fp8_e4m3", "fp8_e5m2"])
@pytest.mark.parametrize("scale", [0.037, 2.0 ** -140, 1e30])
def test_cast_transpose(rows, cols, fmt, scale):
    import voyager_b200 as vb

    x = C.randn(rows + cols, rows, cols, outliers=0.01)
    x.view(-1)[::53] *= 2.0 ** -118
    x.view(-1)[::101] *= -0.0
    s = torch.tensor(scale, dtype=torch.float32).cuda()
    codes, transpose, amax = vb.fp8.quantize_fp8_transpose(x.cuda(), s, fmt)
    padded = torch.zeros(-(-rows * cols // 16) * 16, dtype=torch.bfloat16)
    padded[: rows * cols] = x.reshape(-1)
    want = vb.fp8.quantize_fp8(padded.cuda(), s, fmt)[: rows * cols].view(rows, cols)
    assert torch.equal(codes, want) and torch.equal(transpose, want.T)
    assert float(amax) == float(x.abs().max()) and amax.dim() == 0
    heads = 2
    if cols % 16 == 0:
        heads_t = vb.fp8.transpose_quantize_fp8(x.cuda().view(rows, heads, cols // heads), s, fmt)
        assert torch.equal(heads_t.view(cols, rows), want.T)
