"""The one-elimination factor of the inverse Hessian, and the sweep's kernels at odd block widths."""

import math

import pytest
import torch

from golden_io import bits_equal, describe_mismatch
from oracle import gptq as OG
from oracle import tables as OT

pytestmark = pytest.mark.gpu


def _hessian(k, tokens, seed):
    g = torch.Generator().manual_seed(seed)
    x = 0.7 * torch.randn(tokens, k, generator=g) + 0.3 * (
        torch.randn(tokens, 8, generator=g) @ torch.randn(8, k, generator=g)) / math.sqrt(8)
    return x.T @ x


@pytest.mark.parametrize("k", [1, 7, 128, 130, 384, 1000])
def test_factor_against_float64(k):
    import voyager_b200 as vb

    tokens = 2 * k + 16
    h = _hessian(k, tokens, k)
    got = vb.gptq.hessian_inverse_chol(h.cuda(), tokens, 0.01).cpu().double()
    want = OG.hessian_inverse_chol(h.double(), tokens, 0.01)
    lib = OG.hessian_inverse_chol(h.clone(), tokens, 0.01).double()   # factor, invert, factor in float32
    scale = want.abs().max()
    err, lib_err = float((got - want).abs().max() / scale), float((lib - want).abs().max() / scale)
    assert torch.equal(got, got.triu())
    assert err <= max(2 * lib_err, 1e-6), (err, lib_err)


def test_indefinite_hessians_escalate_or_are_refused():
    import voyager_b200 as vb

    h = _hessian(256, 64, 3)                       # rank 64 of 256
    h -= 0.05 * h.diagonal().mean() * torch.eye(256)
    got = vb.gptq.hessian_inverse_chol(h.cuda(), 64, 0.01).cpu().double()
    want = OG.hessian_inverse_chol(h.double(), 64, 0.01)
    assert float((got - want).abs().max() / want.abs().max()) < 1e-3
    for bad in (-torch.eye(130) * 1e9, torch.full((64, 64), float("nan"))):
        with pytest.raises(torch.linalg.LinAlgError):
            vb.gptq.hessian_inverse_chol(bad.cuda(), 1, 0.01)


@pytest.mark.parametrize("rows,k,bs,affine", [(1, 18, 18, True), (33, 100, 100, True), (17, 24, 24, False), (50, 128, 128, False),
                                              (15, 7, 7, False)])
def test_single_block_of_any_width(rows, k, bs, affine):
    import voyager_b200 as vb

    h = _hessian(k, 512, rows + k)
    hinv = OG.hessian_inverse_chol(h.clone(), 512, 0.01)
    w = torch.randn(rows, k, generator=torch.Generator().manual_seed(k)) * 0.02
    if affine:
        q = OT.quantization_map("uint4")
        want = OG.sweep_affine(w, hinv, q, 0.0, 15.0, bs)
        got = vb.gptq.sweep(w.cuda(), hinv.cuda(), bs, q.cuda(), affine_range=(0.0, 15.0)).cpu()
    else:
        q, s = OT.quantization_map("int4"), OT.quantization_map("fp8_e5m3")
        sal = h.diagonal().clone()
        want = OG.sweep(w, hinv, sal, q, s, 7.0, bs, False)
        got = vb.gptq.sweep(w.cuda(), hinv.cuda(), bs, q.cuda(), s.cuda(), 7.0, sal.cuda(), False).cpu()
    assert bits_equal(got, want), describe_mismatch(got, want)


@pytest.mark.parametrize("rows,k,n", [(1, 132, 4), (130, 260, 128), (300, 1000, 64), (5, 51, 16), (64, 640, 100)])
def test_trailing_update(rows, k, n):
    import voyager_b200 as vb

    N = vb._native
    g = torch.Generator().manual_seed(k)
    work, deltas, u = (torch.randn(*s, generator=g).cuda() for s in ((rows, k), (rows, n), (k, k)))
    got = work.clone()
    N.check(N.lib().vq_gptq_update(got.data_ptr(), deltas.data_ptr(), u.data_ptr(), rows, k, 0, n,
                                   torch.cuda.current_stream().cuda_stream))
    want = work.double()
    want[:, n:] -= deltas.double() @ u[:n, n:].double()
    bound = 4 * math.sqrt(n) * 2.0 ** -24 * (deltas.abs().double() @ u[:n, n:].abs().double()) + 2.0 ** -23 * want[:, n:].abs()
    assert torch.equal(got[:, :n], work[:, :n])
    assert bool(((got[:, n:].double() - want[:, n:]).abs() <= bound).all())
