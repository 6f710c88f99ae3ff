"""The one-kernel attention on prompts that fill no 128-row block, against the separate operators."""

import math

import pytest
import torch

from test_gpu_attention import _eager_bf16_attention, _operands, _separate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,kv,groups", [(8, 1, 1), (120, 2, 2), (136, 1, 4), (264, 2, 3), (776, 2, 4), (1016, 1, 2)])
def test_fp8(T, kv, groups):
    import voyager_b200 as vb

    q, k, vt = _operands(T, kv, groups, T + kv + groups)
    a, b = torch.tensor(0.37).cuda(), torch.tensor(1.0 / 448.0 * 0.9).cuda()
    p_scale = torch.tensor(1.0 / 448.0, dtype=torch.bfloat16).cuda()
    want = _separate(vb, q, k, vt, a, 1 / math.sqrt(128), p_scale, b, T).float()
    # the value rows carry garbage past T, and the next head's queries follow the last block's rows
    padded = torch.full((kv, 128, -(-T // 16) * 16 + 16), 0x7F, dtype=torch.uint8, device="cuda")
    padded[:, :, :T] = vt
    for values in (vt, padded[:, :, :T]):
        got = vb.fp8.attention_fp8(q, k, values, a, 1 / math.sqrt(128), p_scale, b, ragged=True)
        assert vb.fp8.attention_status() == 0
        err = (got.float() - want).abs()
        assert float(err.max()) <= 1e-2 * float(want.abs().max()) and float((err > 0).float().mean()) < 0.05
    scale = (got.float().abs().amax() / 448.0).bfloat16()
    codes = vb.fp8.attention_fp8(q, k, vt, a, 1 / math.sqrt(128), p_scale, b, scale, ragged=True)
    assert torch.equal(codes.view(torch.uint8), vb.fp8.transpose_heads_quantize_fp8(got.view(kv * groups, T, 128), scale))


@pytest.mark.parametrize("T,kv,groups", [(1, 1, 1), (127, 1, 2), (129, 2, 2), (333, 1, 4), (1000, 2, 4)])
def test_bf16(T, kv, groups):
    from voyager_b200 import fp8 as F8

    g = torch.Generator().manual_seed(T + kv + groups)
    q, k, v = ((torch.randn(T, h, 128, generator=g) * s).bfloat16().cuda() for h, s in ((kv * groups, 1.5), (kv, 1.5), (kv, 1.0)))
    got = F8.attention_bf16_heads(q.transpose(0, 1).contiguous(), k.transpose(0, 1).contiguous(), v.permute(1, 2, 0), ragged=True)
    assert F8.attention_status() == 0
    want = _eager_bf16_attention(q, k, v)
    diff = (got.float() - want.float()).abs()
    # as for whole blocks: a probability on a bfloat16 rounding boundary may move by one step
    assert float(diff.max()) <= 2e-2 * float(want.float().abs().max()), float(diff.max())
    assert float(diff.pow(2).mean().sqrt()) <= 2e-3 * float(want.float().pow(2).mean().sqrt())


@pytest.mark.parametrize("T", [8, 24, 776])
def test_padded_value_rows_of_the_projection_cast(T):
    import voyager_b200 as vb

    g = torch.Generator().manual_seed(T)
    qkv = torch.randn(T, 6 * 128, generator=g).bfloat16().cuda()
    q, k, v = (t.unflatten(1, (-1, 128)) for t in (qkv[:, :512], qkv[:, 512:640], qkv[:, 640:]))
    cos, sin = (torch.randn(T, 128, generator=g).bfloat16().cuda() for _ in range(2))
    s = torch.tensor(0.02, dtype=torch.bfloat16).cuda()
    for a, b in zip(vb.fp8.qkv_post_fp8(q, k, v, cos, sin, s, s, s, ragged=True), vb.fp8.qkv_post_fp8(q, k, v, cos, sin, s, s, s)):
        assert torch.equal(a, b)
