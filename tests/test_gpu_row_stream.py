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


def test_captured_call_outlives_a_wider_one():
    """A graph captured for a narrow weight replays correctly after a much wider weight went through the same entry and
    after whatever that call freed was handed out again."""
    import voyager_b200 as vb

    m, k, bs = 3, 2048, 64
    w = _packed(vb, 1000, k, bs, 3)
    x = torch.randn(m, k, generator=torch.Generator(device="cuda").manual_seed(4), device="cuda").bfloat16()
    want = vb.packed.linear_lut4(x, w, out_dtype=torch.float32)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = vb.packed.linear_lut4(x, w, out_dtype=torch.float32)
    wide = _packed(vb, 128256, 256, bs, 5)
    vb.packed.linear_lut4(x[:, :256].contiguous(), wide)
    del wide
    others = [torch.full((1024 * 4,), 7, dtype=torch.int32, device="cuda") for _ in range(64)]   # 16 KB each
    for _ in range(3):
        out.fill_(float("nan"))
        graph.replay()
        assert torch.equal(out, want)
    assert all(bool((t == 7).all()) for t in others)


@pytest.mark.parametrize("packed", [True, False])
def test_two_streams_at_a_time(packed):
    import voyager_b200 as vb

    m, k, bs = 2, 4096, 64
    x = torch.randn(m, k, generator=torch.Generator(device="cuda").manual_seed(6), device="cuda").bfloat16()
    calls = []
    for seed in (7, 8):
        w = _packed(vb, 2000, k, bs, seed)
        if packed:
            calls.append(lambda w=w: vb.packed.linear_lut4(x, w, out_dtype=torch.float32))
        else:
            codes, ones = vb.packed.unpack_lut4_weight(w), torch.ones(m, k // bs, device="cuda").bfloat16()
            calls.append(lambda w=w, codes=codes, ones=ones: torch.ops.quantized_ops.linear_mx(
                x, codes, None, input_scale=ones, weight_scale=w.scale, block_size=bs, weight_code=w.levels,
                out_dtype=torch.float32))
    want = [call() for call in calls]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in calls]
    got = [[], []]
    for _ in range(50):
        for i, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                got[i].append(calls[i]())
    torch.cuda.synchronize()
    for i in range(2):
        assert all(torch.equal(g, want[i]) for g in got[i])


@pytest.mark.parametrize("m,k", [(2, 327680), (32, 153600)])   # 150 slices and more: there are 148 SMs
@pytest.mark.parametrize("packed", [True, False])
def test_more_slices_than_sms(packed, m, k):
    import voyager_b200 as vb

    bs, n = 64, 24
    w = _packed(vb, n, k, bs, 9)
    x = torch.randn(m, k, generator=torch.Generator(device="cuda").manual_seed(10), device="cuda").bfloat16()
    codes = vb.packed.unpack_lut4_weight(w)
    if packed:
        got = vb.packed.linear_lut4(x, w, out_dtype=torch.float32)
    else:
        got = torch.ops.quantized_ops.linear_mx(x, codes, None, input_scale=torch.ones(m, k // bs, device="cuda").bfloat16(),
                                                weight_scale=w.scale, block_size=bs, weight_code=w.levels,
                                                out_dtype=torch.float32)
    vb.ops.gemm_status()
    real = (w.levels[codes.long()].float() * w.scale.float().repeat_interleave(bs, 1)).bfloat16().double()
    # float32 sums of k exact products: random-walk rounding of about sqrt(k) 2^-24 of the terms' size
    bound = 4 * k ** 0.5 * 2.0 ** -24 * (x.double().abs() @ real.abs().T)
    assert bool(((got.double() - x.double() @ real.T).abs() <= bound).all())


def _off(t):
    """The same values two bytes past a 16-byte boundary."""
    flat = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    at = flat[1:t.numel() + 1]
    at.copy_(t.reshape(-1))
    assert at.data_ptr() % 16 == 2
    return at.view(t.shape)


@pytest.mark.parametrize("m", [3, 20])
@pytest.mark.parametrize("n,k,bs", [(40, 4096, 64), (33, 1024, 16)])
@pytest.mark.parametrize("coded", [False, True])
@pytest.mark.parametrize("off", [False, True])
def test_special_scales_and_scales_anywhere(m, n, k, bs, coded, off):
    """Infinite and NaN scales, zero ones beside infinite ones, and scale rows that TMA cannot fetch: the streamed product
    has the read-back path's infinities and NaNs, and its values up to the order of the sums."""
    import voyager_b200 as vb

    g = torch.Generator(device="cuda").manual_seed(m + n)
    a, w = (torch.randint(0, 16, (r, k), generator=g, device="cuda").bfloat16() for r in (m, n))
    sa, sw = ((torch.rand(r, k // bs, generator=g, device="cuda") + 0.5).bfloat16() for r in (m, n))
    a[1], w[1] = 3.0, 9.0       # products of one sign: an infinite scale gives an infinity and not their difference
    sw[1, 2], sw[n - 1, 0], sw[5, 3], sa[2, 1], sa[0, 3] = float("inf"), float("nan"), -float("inf"), float("inf"), 0.0
    levels = torch.linspace(-1, 1, 16, device="cuda").bfloat16() if coded else None
    if off:
        sa, sw = _off(sa), _off(sw)
    layout = vb.ops.LINEAR_LAYOUT
    got = vb.ops._mx_gemm_few_rows(layout, a, w, None, sa, sw, bs, levels, levels, None, layout, torch.float32)
    assert got is not None
    real_a, real_w = (torch.ops.quantized_ops.dequantize_mx(c, s, bs, levels) for c, s in ((a, sa), (w, sw)))
    want = real_a.double() @ real_w.double().T
    assert torch.equal(got.isnan(), want.isnan()) and bool(want.isnan().any()) and bool(want.isinf().any())
    assert torch.equal(got.isinf(), want.isinf()) and torch.equal(got[want.isinf()], want[want.isinf()].float())
    # float32 sums of k exact products: random-walk rounding of about sqrt(k) 2^-24 of the terms' size
    bound = 4 * k ** 0.5 * 2.0 ** -24 * (real_a.double().abs() @ real_w.double().abs().T)
    finite = want.isfinite()
    assert bool(((got.double() - want).abs() <= bound)[finite].all())
    if coded and bs >= 32:
        packed = vb.packed.PackedLUT4Weight(vb.packed.pack_lut4_weight(w, sw, levels, bs).codes, sw, levels, bs)
        again = vb.packed.linear_lut4(a, packed, input_scale=sa, input_code=levels, out_dtype=torch.float32)
        assert torch.equal(again.isnan(), want.isnan()) and torch.equal(again.isinf(), want.isinf())
        assert bool(((again.double() - want).abs() <= bound)[finite].all())


@pytest.mark.parametrize("m", [1, 16, 32])
def test_one_clearing_for_a_step(m):
    """Products on counters cleared together are the products that clear their own, also when captured and replayed."""
    import voyager_b200 as vb

    P = vb.packed
    weights = [_packed(vb, n, k, 64, n) for n, k in ((1000, 2048), (24, 4096), (4096, 1024))]
    xs = [torch.randn(m, w.shape[1], generator=torch.Generator(device="cuda").manual_seed(i), device="cuda").bfloat16()
          for i, w in enumerate(weights)]
    want = [P.linear_lut4(x, w, out_dtype=torch.float32) for x, w in zip(xs, weights)]

    def step():
        return [P.linear_counted(x, w, c, out_dtype=torch.float32) for x, w, c in zip(xs, weights, P.step_counters(weights))]

    assert all(torch.equal(a, b) for a, b in zip(step(), want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    for _ in range(3):
        for t in out:
            t.fill_(float("nan"))
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(out, want))
    counters = P.step_counters(weights)
    for bad in (counters[1], counters[0].float(), counters[0].cpu()):
        with pytest.raises(ValueError):
            P.linear_counted(xs[0], weights[0], bad)
