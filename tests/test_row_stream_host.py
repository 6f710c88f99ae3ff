"""Host side of the weight-streaming linears: workspaces and the cut of the weight."""

import ctypes

import pytest
import torch

import voyager_b200 as vb


def test_scratch_belongs_to_one_call():
    calls = [[t for t in vb.packed._scratch(torch.device("cpu"), 1, n, 4096) if isinstance(t, torch.Tensor)]
             for n in (4096, 4096, 128256)]
    spans = [[(t.data_ptr(), t.data_ptr() + t.numel() * t.element_size()) for t in call] for call in calls]
    for i, one in enumerate(spans):
        for other in spans[:i]:
            assert all(a[1] <= b[0] or b[1] <= a[0] for a in one for b in other)


def _slice(rows, n, k, packed, i):
    values = [ctypes.c_int64() for _ in range(4)]
    vb._native.check(vb._native.lib().vq_row_stream_slice(rows, n, k, packed, i, *map(ctypes.byref, values)), "slice")
    return [v.value for v in values]


@pytest.mark.parametrize("rows", [1, 9, 17, 25])
@pytest.mark.parametrize("packed", [0, 1])
@pytest.mark.parametrize("k", [128, 4096, 14336, 327680, 11_108_352, 16_777_216, 33_554_432, (1 << 30) - 128, (1 << 31) - 128])
def test_slices_cover_the_contraction(rows, packed, k):
    n = 4096 if k < 1 << 24 else 16
    steps, slices, begin, _ = _slice(rows, n, k, packed, 0)
    assert steps == k // (128 if packed else 32) and 1 <= slices <= steps and begin == 0
    # the longest slice that the shared memory holds, in steps
    longest = {(1, 0): 64, (9, 0): 32, (17, 0): 40, (25, 0): 28, (1, 1): 16, (9, 1): 8, (17, 1): 10, (25, 1): 8}[rows, packed]
    picks = range(slices) if slices < 20000 else sorted({0, 1, slices // 3, slices // 2, slices - 2, slices - 1,
                                                         *range(0, slices, slices // 500)})
    for i in picks:
        _, _, begin, end = _slice(rows, n, k, packed, i)
        assert begin == i * steps // slices and end == (i + 1) * steps // slices, i
        assert 1 <= end - begin <= longest
    assert _slice(rows, n, k, packed, slices - 1)[3] == steps


@pytest.mark.parametrize("rows,k", [(32, 58_720_256 + 1024), (8, 134_217_728 + 2048), (1, (1 << 30) - 64)])
def test_too_many_slices_are_left_to_the_gemm(rows, k):
    from torch._subclasses.fake_tensor import FakeTensorMode

    assert vb._native.lib().vq_gemm_mx_rows_workspace_bytes(rows, 16, k) == 0
    assert vb._native.lib().vq_gemm_mx_rows_workspace_bytes(rows, 16, 4096) > 0
    with FakeTensorMode():
        codes = lambda r: torch.empty(r, k, dtype=torch.bfloat16, device="cuda")  # noqa: E731
        scale = lambda r: torch.empty(r, k // 64, dtype=torch.bfloat16, device="cuda")  # noqa: E731
        assert vb.ops._mx_gemm_few_rows(vb.ops.LINEAR_LAYOUT, codes(rows), codes(16), None, scale(rows), scale(16), 64, None,
                                        None, None, vb.ops.LINEAR_LAYOUT, torch.float32) is None


def _route(rows, n, k, bs, lookup):
    """What linear_mx's few-rows path makes of a call: None where it leaves it to the GEMM."""
    from torch._subclasses.fake_tensor import FakeTensorMode

    with FakeTensorMode():
        make = lambda *shape: torch.empty(*shape, dtype=torch.bfloat16, device="cuda")  # noqa: E731
        levels = make(16) if lookup else None
        try:
            return vb.ops._mx_gemm_few_rows(vb.ops.LINEAR_LAYOUT, make(rows, k), make(n, k), None, make(rows, k // bs),
                                            make(n, k // bs), bs, levels, levels, None, vb.ops.LINEAR_LAYOUT, torch.bfloat16)
        except RuntimeError:   # it went on to the kernel, which takes no tensor without memory
            return "streamed"


@pytest.mark.parametrize("rows,n,k,lookup,streamed", [
    (1, 128256, 4096, True, True), (24, 128256, 4096, True, True), (24, 18944, 4096, False, True), (24, 512, 128, False, True),
    (25, 8448, 4096, True, True), (32, 10240, 5120, True, True), (32, 14336, 4096, True, False), (25, 22016, 4096, True, False),
    (32, 12288, 10752, True, True), (32, 14336, 4096, False, True), (32, 18944, 4096, False, False),
    (32, 22016, 4096, False, True), (25, 37888, 4096, False, False), (32, 128256, 4096, False, False), (33, 512, 512, False, False)])
def test_which_products_are_streamed(rows, n, k, lookup, streamed):
    assert (_route(rows, n, k, 64, lookup) is not None) == streamed
