"""The inverse's factor from Hessians that are not one dense row-major symmetric matrix."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _hessian(k):
    g = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn(2 * k + 16, k, generator=g, device="cuda")
    h = x.T @ x
    return (h + h.T) / 2      # equal triangles to the last bit


@pytest.mark.parametrize("k", [5, 128, 200, 512])
def test_strides_do_not_matter(k):
    import voyager_b200 as vb

    h = _hessian(k)
    want = vb.gptq.hessian_inverse_chol(h, 7, 0.01)
    wide = torch.zeros(k, k + 3, device="cuda")
    wide[:, 1:k + 1] = h
    for other in (h.T.contiguous().T, wide[:, 1:k + 1], wide[:, 1:k + 1].T):
        assert torch.equal(vb.gptq.hessian_inverse_chol(other, 7, 0.01), want)
    # the whole solve on a Hessian stored by columns
    w = torch.randn(16, k, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda") * 0.02
    q = vb.get_quantization_map("uint4", "cuda")
    solve = lambda hessian: vb.gptq.compensate_weight_affine(w, hessian, 7, q, 0.0, 15.0, min(k, 128), 0.01)  # noqa: E731
    assert torch.equal(solve(h.T.contiguous().T), solve(h))


@pytest.mark.parametrize("k", [5, 128, 200])
def test_only_the_lower_triangle_is_read(k):
    import voyager_b200 as vb

    h = _hessian(k)
    want = vb.gptq.hessian_inverse_chol(h, 7, 0.01)
    half = h.tril() + torch.full_like(h, 1e6).triu(1)
    assert torch.equal(vb.gptq.hessian_inverse_chol(half, 7, 0.01), want)
