"""linear_mx of a few rows, streamed from the operator's storage, against float64 and against the read-back path."""

import pytest
import torch

from oracle import quantizers as OQ

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 7, 8, 9, 16, 17, 24, 31, 32])
@pytest.mark.parametrize("n,k,bs,coded", [(1, 32, 8, False), (33, 96, 32, True), (4096, 1024, 16, False), (1000, 4160, 64, True),
                                          (72, 8192, 128, True), (513, 544, 16, False)])
def test_few_rows(m, n, k, bs, coded):
    import voyager_b200 as vb

    g = torch.Generator().manual_seed(m + n + k)
    pick = lambda *s: torch.randint(0, 16, s, generator=g).bfloat16() if coded else torch.randint(-127, 128, s, generator=g).bfloat16()  # noqa: E731
    ca, cw = pick(m, k), pick(n, k)
    if coded and k > 64:
        cw[0, 3], cw[-1, 5], ca[0, 2] = -3.0, 7.5, -1.0   # the operator truncates, and wraps a negative index once
    sa, sw = (torch.rand(r, k // bs, generator=g).bfloat16() + 0.5 for r in (m, n))
    levels = torch.sort(torch.randn(16, generator=g)).values.bfloat16() if coded else None
    bias, alpha = torch.randn(n, generator=g).bfloat16(), torch.tensor(0.75)
    dev = lambda t: None if t is None else t.cuda()  # noqa: E731
    kw = dict(input_scale=sa.cuda(), weight_scale=sw.cuda(), block_size=bs, input_code=dev(levels), weight_code=dev(levels))
    got = torch.ops.quantized_ops.linear_mx(ca.cuda(), cw.cuda(), None, out_dtype=torch.float32, **kw)
    assert vb.ops._mx_gemm_few_rows("xc,kc->xk", ca.cuda(), cw.cuda(), None, kw["input_scale"], kw["weight_scale"], bs,
                                    kw["input_code"], kw["weight_code"], None, "xc,kc->xk", torch.float32) is not None
    a = OQ.dequantize_mx(ca, sa, bs, code=levels).double()
    w = OQ.dequantize_mx(cw, sw, bs, code=levels).double()
    # float32 sums of k exact products: random-walk rounding of about sqrt(k) 2^-24 of the terms' size
    bound = 4 * k ** 0.5 * 2.0 ** -24 * (a.abs() @ w.abs().T)
    assert bool(((got.cpu().double() - a @ w.T).abs() <= bound).all())
    full = torch.ops.quantized_ops.linear_mx(ca.cuda(), cw.cuda(), bias.cuda(), alpha=alpha.cuda(), **kw)
    want = (a @ w.T * 0.75 + bias.double())
    assert full.dtype == torch.bfloat16
    assert bool(((full.cpu().double() - want).abs() <= 2.0 ** -8 * want.abs() + 2 * bound).all())
