"""The FP8 cast with its transpose where the transposed rows begin at any byte, and around the tiles' edges."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 2, 3, 5, 126, 127, 128, 129, 130, 131, 132, 144, 255, 258, 777])
@pytest.mark.parametrize("heads,d", [(1, 8), (3, 64), (2, 136)])
@pytest.mark.parametrize("dtype", ["fp8_e4m3", "fp8_e5m2"])
def test_rows_that_begin_anywhere(T, heads, d, dtype):
    import voyager_b200 as vb

    x = torch.randn(T, heads, d, generator=torch.Generator(device="cuda").manual_seed(T + d), device="cuda").bfloat16()
    scale = torch.tensor(0.013, dtype=torch.bfloat16, device="cuda")
    # the plain cast takes multiples of 16 elements
    padded = torch.nn.functional.pad(x, (0, 0, 0, 0, 0, T % 2))
    want = vb.fp8.quantize_fp8(padded, scale, dtype).view(torch.uint8)[:T]
    got = vb.fp8.transpose_quantize_fp8(x, scale, dtype)
    assert torch.equal(got.view(torch.uint8), want.permute(1, 2, 0))
    # both layouts of a matrix, the maximum beside them, and nothing written outside the rows
    m = x.view(T, heads * d)
    codes, transpose, amax = vb.fp8.quantize_fp8_transpose(m, scale, dtype)
    assert torch.equal(codes.view(torch.uint8), want.reshape(T, heads * d))
    assert torch.equal(transpose.view(torch.uint8), want.reshape(T, heads * d).T)
    assert torch.equal(amax.float(), m.float().abs().amax())


@pytest.mark.parametrize("T", [2, 7, 129, 130, 255])
def test_nothing_is_written_beside_the_rows(T):
    import voyager_b200 as vb

    N = vb._native
    x = torch.randn(T, 1, 16, generator=torch.Generator(device="cuda").manual_seed(T), device="cuda").bfloat16()
    scale = torch.tensor(0.02, device="cuda")
    buffer = torch.full((16 * T + 64,), 0xAA, dtype=torch.uint8, device="cuda")
    N.check(N.lib().vq_transpose_quantize_fp8(x.data_ptr(), buffer.data_ptr() + 32, None, None, N.IN_E4M3, T, 1, 16, 16,
                                              scale.data_ptr(), 2, torch.cuda.current_stream().cuda_stream))
    assert bool((buffer[:32] == 0xAA).all()) and bool((buffer[32 + 16 * T:] == 0xAA).all())
    want = vb.fp8.transpose_quantize_fp8(x, scale).view(torch.uint8)
    assert torch.equal(buffer[32:32 + 16 * T].view(16, T), want[0])
