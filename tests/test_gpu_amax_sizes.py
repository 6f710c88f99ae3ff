"""The tensor maximum over sizes on both sides of one load a thread, and codebook read-backs around the table's threshold."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# a grid of 592 blocks of 256 threads, eight values a load
@pytest.mark.parametrize("n", [1, 8, 2047, 2048, 592 * 2048 - 8, 592 * 2048, 592 * 2048 + 8, 2 * 592 * 2048 + 16, 4 * 592 * 2048 + 9,
                               5 * 592 * 2048 - 1])
@pytest.mark.parametrize("where", [0.0, 0.4999, 1.0])
def test_amax_finds_the_largest_anywhere(n, where):
    import voyager_b200 as vb

    N = vb._native
    x = torch.full((n,), -0.5, device="cuda").bfloat16()
    at = min(int(n * where), n - 1)
    out = torch.zeros((), device="cuda")
    for value in (-3.25, float("-inf"), float("nan")):
        x[at] = value
        out.zero_()
        N.check(N.lib().vq_amax(x.data_ptr(), 0, n, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
        want = x[at].abs().float()
        assert torch.equal(out, want) or (bool(out.isnan()) and bool(want.isnan()))


@pytest.mark.parametrize("rows,cols", [(1, 64), (15, 4096), (16, 4096), (31, 2112), (32, 2112)])
def test_read_back_through_a_codebook(rows, cols):
    import voyager_b200 as vb

    g = torch.Generator(device="cuda").manual_seed(rows)
    codes = torch.randint(0, 16, (rows, cols), generator=g, device="cuda")
    levels = torch.randn(16, generator=g, device="cuda").bfloat16()
    scale = torch.randn(rows, cols // 64, generator=g, device="cuda").bfloat16()
    got = torch.ops.quantized_ops.dequantize_mx(codes.bfloat16(), scale, 64, levels)
    assert torch.equal(got, levels[codes] * scale.repeat_interleave(64, 1))
