"""The packed decode linear where its even cut of the weight falls inside tiles: between warps, CTAs and K slices."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 24, 25, 32])
@pytest.mark.parametrize("n,k,bs", [(1, 128, 32), (33, 5248, 64), (6144, 1152, 64), (4100, 4096, 128), (72, 16512, 128)])
def test_against_float64(m, n, k, bs):
    import voyager_b200 as vb

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    levels = torch.linspace(-1, 1, 16, device="cuda").bfloat16()
    codes = torch.randint(0, 16, (n, k), generator=g, device="cuda").bfloat16()
    scale = (torch.rand(n, k // bs, generator=g, device="cuda") + 0.5).bfloat16()
    x = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    packed = vb.packed.pack_lut4_weight(codes, scale, levels, bs)
    got = vb.packed.linear_lut4(x, packed, out_dtype=torch.float32)
    w = (levels[codes.long()].float() * scale.float().repeat_interleave(bs, 1)).bfloat16().double()
    want = x.double() @ w.T
    # float32 sums of k exact products: random-walk rounding of about sqrt(k) 2^-24 of the terms' size
    bound = 4 * k ** 0.5 * 2.0 ** -24 * (x.double().abs() @ w.abs().T)
    assert bool(((got.double() - want).abs() <= bound).all())
    assert torch.equal(got, vb.packed.linear_lut4(x, packed, out_dtype=torch.float32))
