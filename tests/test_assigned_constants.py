"""Arrays that a caller assigns to a quantizer stay the caller's: what is written into them later reaches the next call."""
import numpy as np
import pytest

import turboquant_plus_b200 as tq


@pytest.mark.parametrize("name", ["rotation", "centroids", "S"])
def test_writes_into_an_assigned_array_are_seen(name):
    holder = tq.QJL(16, seed=1) if name == "S" else tq.PolarQuant(16, 3, seed=1)
    mine = np.array(holder._const.get(name))
    setattr(holder, name, mine)
    uploaded = holder._const.snapshot()
    assert holder._const.same(uploaded)
    mine *= -1.0
    assert not holder._const.same(uploaded)


@pytest.mark.gpu
@pytest.mark.parametrize("name,factor", [("rotation", -1.0), ("centroids", 1.25), ("S", -1.0)])
def test_results_follow_an_assigned_array(name, factor):
    import torch
    x = torch.randn((40, 64), device="cuda", dtype=torch.float64)
    t, fresh = tq.TurboQuant(64, 3, seed=1), tq.TurboQuant(64, 3, seed=1)
    holder = t.qjl if name == "S" else t.polar_quant
    mine = np.array(holder._const.get(name))                # (the attribute itself is not read: that counts as lending)
    setattr(holder, name, mine)
    before = t.quantize(x)
    mine *= factor
    if name == "rotation":
        mine[0] *= -1.0                                     # (both signs of R alone code alike up to ties)
    setattr(fresh.qjl if name == "S" else fresh.polar_quant, name, mine.copy())
    code, want = t.quantize(x), fresh.quantize(x)
    assert torch.equal(code.mse_indices, want.mse_indices) and torch.equal(code.qjl_signs, want.qjl_signs)
    assert not (torch.equal(code.mse_indices, before.mse_indices) and torch.equal(code.qjl_signs, before.qjl_signs))
    assert torch.allclose(t.dequantize(code), fresh.dequantize(want), rtol=1e-12, atol=1e-12)
