"""The weight-streaming linears' tile counters and workspaces: what one call leaves must not reach another."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _packed(vb, n, k, bs, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    levels = torch.linspace(-1, 1, 16, device="cuda").bfloat16()
    codes = torch.randint(0, 16, (n, k), generator=g, device="cuda").bfloat16()
    scale = (torch.rand(n, k // bs, generator=g, device="cuda") + 0.5).bfloat16()
    return vb.packed.pack_lut4_weight(codes, scale, levels, bs)


def test_counters_hold_anything_before_a_call():
    """A launch that gave up waiting leaves tiles counted in part; the next call must not see that."""
    import voyager_b200 as vb

    m, n, k, bs = 4, 520, 4096, 64
    w = _packed(vb, n, k, bs, 1)
    x = torch.randn(m, k, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda").bfloat16()
    want = vb.packed.linear_lut4(x, w, out_dtype=torch.float32)
    lib = vb._native.lib()
    work = torch.empty(int(lib.vq_gemm_lut4_workspace_floats(m, n, k)), device="cuda")
    counters = torch.full((int(lib.vq_gemm_lut4_counters(n)),), 1, dtype=torch.int32, device="cuda")
    for left in (1, 3, -1):
        counters.fill_(left)
        out = torch.full((m, n), float("nan"), device="cuda")
        vb._native.check(lib.vq_gemm_lut4(x.data_ptr(), k, None, None, 0, m, w.codes.data_ptr(), w.scale.data_ptr(),
                                          w.levels.data_ptr(), bs, out.data_ptr(), 2, n, k, None, 0, None, 0,
                                          work.data_ptr(), counters.data_ptr(), torch.cuda.current_stream().cuda_stream),
                         "vq_gemm_lut4")
        assert torch.equal(out, want)
