"""Host arrays of several MB to the GPU and back under torch's modes: the threads that help with a large copy do not have the
caller's modes, and tensors made under inference mode refuse to be written to outside it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["inference_mode", "no_grad"])
def test_large_arrays_under_a_mode(mode):
    import torch
    import turboquant_plus_b200 as tq
    rng = np.random.default_rng(1)
    x = rng.standard_normal((40000, 128)).astype(np.float32)
    quantizer = tq.TurboQuantMSE(128, 3, seed=1)
    idx, norms = quantizer.quantize(x)
    back = quantizer.dequantize(idx, norms)
    with getattr(torch, mode)():
        for _ in range(20):                          # whether a helper gets a piece depends on timing
            i, n = quantizer.quantize(x)
            assert np.array_equal(i, idx) and np.array_equal(n, norms)
            assert np.array_equal(quantizer.dequantize(i, n), back)
