"""What the decode attention kernel hands back to the caller's operators, and what it refuses."""

import pytest
import torch

import voyager_b200 as vb


def _call(R, off, out):
    """The entry on real memory of the calling process; every case here returns before the launch."""
    lib = vb._native.lib()
    p = out.data_ptr()
    return lib.vq_kivi_decode_attention(p, p, p, p, p, p, p, p + off, p + off, p, 1, 4, 64, R, 128, 64, 64, 1.0, None)


@pytest.mark.parametrize("R,off,want", [(53, 2, -3), (17, 8, -3), (127, 14, -3),    # ragged and misaligned: not taken
                                        (64, 2, -1), (128, 8, -1),                  # whole tiles, misaligned: an error
                                        (7, 0, -3), (7, 2, -3)])                    # fewer than 16 positions: not taken
def test_misaligned_windows(R, off, want):
    buffer = torch.zeros(4096, dtype=torch.float64)
    assert buffer.data_ptr() % 16 == 0
    assert _call(R, off, buffer) == want


@pytest.mark.gpu
def test_a_misaligned_ragged_window_runs_the_operators():
    t = {n: vb.get_quantization_map(n, "cuda") for n in ("uint2", "fp8_e4m3")}
    g = torch.Generator(device="cuda").manual_seed(0)
    kv = lambda n: torch.randn(1, 2, n, 128, generator=g, device="cuda").bfloat16()  # noqa: E731
    keys = vb.kivi.quantize_cache(kv(128), t["uint2"], -2, 64, 2, t["fp8_e4m3"])
    values = vb.kivi.quantize_cache(kv(128), t["uint2"], -1, 64, 2, t["fp8_e4m3"])
    q = torch.randn(1, 2, 4, 128, generator=g, device="cuda").bfloat16()
    flat = torch.randn(2 * 53 * 128 + 1, generator=g, device="cuda").bfloat16()
    window = flat[1:].view(1, 2, 53, 128)
    assert window.data_ptr() % 16 == 2
    assert vb.kivi.decode_attention(q, keys, values, window, window) is None
    assert vb.kivi.decode_attention(q, keys, values, window.clone(), window.clone()) is not None
