"""The tensor maximum over sizes on both sides of one load a thread."""

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
