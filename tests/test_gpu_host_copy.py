"""Host arrays to the GPU and back through the staging pieces: sizes around one piece, around the 2 MB page pieces and around
the number of buffers, arrays that do not start on an element boundary of a page, every pair of types the classes use."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [0, 1, 32768, 32769, 262143, 262145, 300001, 4 * 262144 + 7, 40 * 262144 + 1]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("host,dev", [("int64", "uint8"), ("float64", "float64"), ("float32", "float32"), ("float64", "float32"),
                                      ("int8", "int8"), ("float16", "float16"), ("float16", "float32")])
def test_there_and_back(host, dev, n):
    import torch
    import turboquant_plus_b200._native as nv
    rng = np.random.default_rng(n)
    src = rng.integers(0, 16, n).astype(host) if "int" in host else rng.standard_normal(n).astype(host)
    code = {"uint8": -2, "int8": -3, "float16": nv.F16, "float32": nv.F32, "float64": nv.F64}[dev]
    for offset in (0, 5):                                    # the second: a slice that starts inside a larger array
        base = np.empty(n + 8, host)
        base[offset:offset + n] = src
        t = nv.host().upload(base[offset:offset + n], 0, code)
        assert t.dtype == getattr(torch, dev) and np.array_equal(t.cpu().numpy(), src.astype(dev))
        small = torch.arange(3, device="cuda", dtype=torch.float32)
        out, extra = np.full(n + 8, 7, host), np.empty(3, np.float64)
        nv.host().download(t, out[offset:offset + n], small, extra)
        assert np.array_equal(out[offset:offset + n], src.astype(dev).astype(host))
        assert (out[:offset] == 7).all() and (out[offset + n:] == 7).all() and np.array_equal(extra, [0, 1, 2])
