"""The vectorised read-back of 16-entry lookup operands equals the operator's arithmetic bit for bit."""

import pytest
import torch

import cases as C
from oracle import quantizers as OQ

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,block", [(1, 64, 64), (3, 320, 64), (7, 1032, 8), (129, 4096, 64), (33, 240, 24)])
@pytest.mark.parametrize("odd", [False, True])
def test_codebook_read_back(rows, k, block, odd):
    import voyager_b200  # noqa: F401

    g = torch.Generator().manual_seed(rows + k)
    codes = torch.randint(0, 16, (rows, k), generator=g).bfloat16()
    if odd:   # values that are no index: the operator truncates, wraps a negative once and clamps
        where = torch.rand(rows, k, generator=g) < 0.05
        codes = torch.where(where, C.randn(3, rows, k) * 12, codes)
    scale = (torch.rand(rows, k // block, generator=g) * 2 ** torch.randint(-130, 20, (rows, k // block), generator=g)).bfloat16()
    levels = C.randn(5, 16)
    want = OQ.dequantize_mx(codes.clamp(-15.9, 15.9), scale, block, code=levels)
    got = torch.ops.quantized_ops.dequantize_mx(codes.clamp(-15.9, 15.9).cuda(), scale.cuda(), block, code=levels.cuda())
    assert torch.equal(got.cpu().view(torch.int16), want.view(torch.int16))
