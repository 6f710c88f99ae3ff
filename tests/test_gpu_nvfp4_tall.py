"""The two-way NVFP4 casts of a matrix with more row tiles than a grid's second extent holds."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("square", [False, True])
def test_more_than_four_million_rows(square):
    import voyager_b200 as vb

    base = torch.randn(128, 64, generator=torch.Generator(device="cuda").manual_seed(0), device="cuda").bfloat16()
    times = 32769                                   # 65538 tiles of 64 rows
    cast = vb.nvfp4.quantize_nvfp4_square if square else vb.nvfp4.quantize_nvfp4_pair
    want, got = cast(base), cast(base.repeat(times, 1))
    codes, scales, codes_t, scales_t, t = (0, 1, 2, 3, 4) if square else (0, 1, 3, 4, 2)
    # one tile repeats: codes along the rows, scales as whole 512-byte tiles
    assert torch.equal(got[t], want[t])
    assert torch.equal(got[codes].view(times, -1), want[codes].view(1, -1).expand(times, -1))
    assert torch.equal(got[codes_t].view(64, times, -1), want[codes_t].view(64, 1, -1).expand(-1, times, -1))
    for s in (scales, scales_t):
        assert torch.equal(got[s].view(times, -1), want[s].view(1, -1).expand(times, -1))
