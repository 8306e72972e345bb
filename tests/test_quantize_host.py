"""Host side of the quantizers."""
import pytest
import torch

from rwkv_quant_b200 import quantize as q


def test_scale_factors_do_not_follow_the_default_type():
    """They are kept per device for the process, and the kernel reads 32-bit floats."""
    q._factors.cache_clear()
    torch.set_default_dtype(torch.float64)
    try:
        kept = [q._factors(s, torch.device("cpu")) for s in (True, False)]
    finally:
        torch.set_default_dtype(torch.float32)
        q._factors.cache_clear()
    assert all(t.dtype == torch.float32 for t in kept)
    assert torch.equal(kept[0], torch.linspace(0.7, 1.15, 19)) and torch.equal(kept[1], torch.ones(1))


@pytest.mark.gpu
@pytest.mark.parametrize("call,bits", [(q.quantize_sb6, 3), (q.quantize_sb6, 7), (q.quantize_sym, 4), (q.quantize_sym, 7)])
def test_bit_widths_are_refused_by_the_library(cuda_lib, call, bits):
    from rwkv_quant_b200._lib import RwkvqError
    w = torch.randn(4, 256, device="cuda")
    with pytest.raises(RwkvqError, match="bits"):
        call("w", "proj", w, bits)
