"""The NVFP4 casts of a training step in two passes equal the operators they stand for, byte for byte."""

import pytest
import torch

import cases as C

pytestmark = pytest.mark.gpu


def _composite(vb, x, axis, seed=None, hadamard=None):
    """quantize_nvfp4 as its operators: rotate, global scale, quantize_mx, pack."""
    if hadamard is not None:
        x = vb.ops.hadamard_rotate(x, axis, hadamard)
    t = vb.calculate_global_scale(x, 6.0, 448.0)
    e2m1, e4m3 = (vb.get_quantization_map(n, "cuda") for n in ("fp4_e2m1", "fp8_e4m3"))
    table = e2m1 if seed is None else vb.formats.qmap_levels(e2m1)
    scale, values = torch.ops.quantized_ops.quantize_mx(x, table, [axis], 16, 6.0, False, e4m3, None, seed, t)
    rows = values.movedim(axis, -1).contiguous()
    packed = vb.nvfp4.pack_nvfp4(rows, scale.movedim(axis, -1).contiguous(), check=False)
    return packed.codes, packed.scales.reshape(-1), t


def _composite_square(vb, w):
    n, k = w.shape
    t = vb.calculate_global_scale(w, 6.0, 448.0)
    amax = w.abs().view(n // 16, 16, k // 16, 16).amax((1, 3))
    e2m1, e4m3 = (vb.get_quantization_map(x, "cuda") for x in ("fp4_e2m1", "fp8_e4m3"))
    scale = torch.ops.quantized_ops.vmap((amax / 6.0 / t).clamp(max=448.0), e4m3)
    scale = torch.where(scale > 0, scale, torch.ones_like(scale))
    values = torch.ops.quantized_ops.quantize(w, scale * t, None, [0, 1], 16, e2m1)
    a = vb.nvfp4.pack_nvfp4(values, scale.repeat_interleave(16, 0), check=False)
    b = vb.nvfp4.pack_nvfp4(values.mT.contiguous(), scale.mT.repeat_interleave(16, 0).contiguous(), check=False)
    return a.codes, a.scales.reshape(-1), b.codes, b.scales.reshape(-1), t


def _input(rows, cols, kind):
    x = C.randn(rows + cols, rows, cols, outliers=0.002).float()
    g = torch.Generator().manual_seed(rows)
    if kind == "special":      # zero blocks, infinities and NaN
        x[:, 16:32] = 0
        x[:16, :16] = 0
        x = torch.where(torch.rand(rows, cols, generator=g) < 1e-4, torch.full((), float("inf")), x)
        x[3, 5] = float("nan")
    elif kind == "tiny":
        x = x * 2.0 ** -126
    elif kind == "wide":
        x = x * torch.exp2(torch.randint(-40, 40, (rows, cols), generator=g).float())
    return x.bfloat16().cuda()


def _same(got, want):
    for a, b in zip(got, want):
        a, b = a.reshape(-1), b.reshape(-1)
        if a.dtype == torch.bfloat16:
            a, b = a.view(torch.int16), b.view(torch.int16)
        assert torch.equal(a, b)


@pytest.mark.parametrize("rows,cols", [(64, 64), (128, 192), (192, 320), (64, 4096), (640, 128)])
@pytest.mark.parametrize("kind", ["plain", "special", "tiny", "wide"])
def test_pair_and_square(rows, cols, kind):
    import voyager_b200 as vb

    x = _input(rows, cols, kind)
    matrix = vb.ops.hadamard_matrix("cuda")
    s0, s1 = (torch.tensor(s, dtype=torch.int64, device="cuda") for s in (11, -7))
    assert vb.nvfp4._two_way(x)
    for seed, seed_t in ((None, None), (s0, None), (None, s1), (s0, s1)):
        for h in (None, matrix):
            got = vb.nvfp4.quantize_nvfp4_pair(x, seed, seed_t, h)
            want = (*_composite(vb, x, -1, seed), *_composite(vb, x.mT.contiguous(), -1, seed_t, h))
            _same(got, want)
    _same(vb.nvfp4.quantize_nvfp4_square(x), _composite_square(vb, x))
    _same(vb.nvfp4.quantize_nvfp4(x), _composite(vb, x, -1))


def test_sixteen_byte_aligned_views():
    import voyager_b200 as vb

    x = _input(128, 192, "plain")
    odd = torch.empty(x.numel() + 8, dtype=x.dtype, device="cuda")[8:].view(x.shape).copy_(x)
    assert odd.data_ptr() % 32 == 16
    _same(vb.nvfp4.quantize_nvfp4_pair(odd), vb.nvfp4.quantize_nvfp4_pair(x))
    _same(vb.nvfp4.quantize_nvfp4(odd), vb.nvfp4.quantize_nvfp4(x))


@pytest.mark.parametrize("n", [8, 1000, 4096 * 33 + 8])
def test_amax_of_bfloat16(n):
    import voyager_b200 as vb

    x = C.randn(n, n, outliers=0.002).cuda()
    assert float(vb.tensor_amax(x)) == float(x.abs().max())
    x[n // 2] = float("nan")
    assert bool(vb.tensor_amax(x).isnan())
