"""FP8 attention, its value rows and the layer on prompts whose length is no multiple of 8 (or is 1)."""

import math

import pytest
import torch
import torch.nn.functional as F

from oracle import layers as OL
from test_gpu_attention import _operands, _separate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,kv,groups", [(1, 1, 1), (7, 2, 2), (127, 1, 3), (129, 2, 1), (333, 2, 4)])
def test_fp8(T, kv, groups):
    import voyager_b200 as vb

    q, k, vt = _operands(T, kv, groups, T + kv + groups)
    a, b = torch.tensor(0.37).cuda(), torch.tensor(1.0 / 448.0 * 0.9).cuda()
    p_scale = torch.tensor(1.0 / 448.0, dtype=torch.bfloat16).cuda()
    # the separate kernels take multiples of 8: positions added behind the prompt are masked for all of its own rows
    Tp = -(-T // 8) * 8
    want = _separate(vb, F.pad(q.view(kv, groups, T, 128), (0, 0, 0, Tp - T)).reshape(kv, groups * Tp, 128),
                     F.pad(k, (0, 0, 0, Tp - T)), F.pad(vt, (0, Tp - T)), a, 1 / math.sqrt(128), p_scale, b, Tp)
    want = want.view(kv, groups, Tp, 128)[:, :, :T].reshape(kv, groups * T, 128).float()
    # NaN bytes from the first one past T, in rows of the caller's and (vt) in rows that the call pads itself
    padded = torch.full((kv, 128, -(-T // 16) * 16 + 16), 0x7F, dtype=torch.uint8, device="cuda")
    padded[:, :, :T] = vt
    for values in (vt, padded[:, :, :T]):
        got = vb.fp8.attention_fp8(q, k, values, a, 1 / math.sqrt(128), p_scale, b, ragged=True)
        assert vb.fp8.attention_status() == 0
        err = (got.float() - want).abs()
        # as for prompts of whole multiples of 8: a probability's code on a rounding boundary may move
        assert float(err.max()) <= 1e-2 * float(want.abs().max()) and float((err > 0).float().mean()) < 0.05
    scale = (got.float().abs().amax() / 448.0).bfloat16()
    codes = vb.fp8.attention_fp8(q, k, vt, a, 1 / math.sqrt(128), p_scale, b, scale, ragged=True)
    assert torch.equal(codes.view(torch.uint8), vb.fp8.transpose_heads_quantize_fp8(got.view(kv * groups, T, 128), scale))


@pytest.mark.parametrize("T", [1, 7, 127, 129, 333])
def test_value_rows_of_the_projection_cast(T):
    import voyager_b200 as vb

    g = torch.Generator().manual_seed(T)
    qkv = torch.randn(T, 6 * 128, generator=g).bfloat16().cuda()
    q, k, v = (t.unflatten(1, (-1, 128)) for t in (qkv[:, :512], qkv[:, 512:640], qkv[:, 640:]))
    cos, sin = (torch.randn(T, 128, generator=g).bfloat16().cuda() for _ in range(2))
    s = torch.tensor(0.02, dtype=torch.bfloat16).cuda()
    got = vb.fp8.qkv_post_fp8(q, k, v, cos, sin, s, s, s, ragged=True)
    want = (vb.fp8.rope_quantize_fp8(q, cos, sin, s), vb.fp8.rope_quantize_fp8(k, cos, sin, s),
            vb.fp8.transpose_quantize_fp8(v, s))
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))


@pytest.mark.parametrize("T", [1, 7, 333])
@pytest.mark.parametrize("merge_qkv", [True, False])
def test_layer(T, merge_qkv):
    import voyager_b200 as vb

    W = vb.workloads
    shape = W.LlamaShape(hidden=512, heads=4, kv_heads=2, head_dim=128, intermediate=1024, vocab=1024)
    params, hidden = W.make_layer_params(0, shape), W.make_hidden_states(1, T, shape)
    scales = W.calibrate_fp8_scales(hidden, params, shape)
    want = OL.fp8_decoder_layer(hidden, params, scales, shape, W.rope_tables(T, shape, "cpu"), W.causal_mask(T, "cpu")).float()
    layer = W.Fp8DecoderLayer({k: v.cuda() for k, v in params.items()}, {k: v.cuda() for k, v in scales.items()}, shape,
                              merge_qkv=merge_qkv)
    got = layer(hidden.cuda()).float().cpu()
    vb.ops.gemm_status()
    assert vb.fp8.attention_status() == 0
    assert float((got - want).norm() / want.norm()) <= 2e-2    # the layers' tolerance against the converted graph
