"""The native host path: inputs that need converting give what converted inputs give, quantizer arrays that a caller
changes take effect, and wrong arguments raise."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cache(torch, tq, hkv=2, **kw):
    cache = tq.PagedKVCache(128, hkv, 4, **kw)
    g = torch.Generator(device="cuda").manual_seed(1)
    k = torch.randn((150, hkv, 128), generator=g, device="cuda").half()
    v = torch.randn((150, hkv, 128), generator=g, device="cuda").half()
    return cache, k, v, torch.randn((1, 4 * hkv, 128), generator=g, device="cuda").half()


def test_converted_arguments():
    import torch
    import turboquant_plus_b200 as tq
    a, k, v, q = _cache(torch, tq)
    b = _cache(torch, tq)[0]
    slots = torch.arange(150, device="cuda") + 128
    a.append(k, v, slots)
    wide = torch.stack([k, v], dim=1)                               # rows that are not contiguous, slots on the host
    b.append(wide[:, 0], wide[:, 1], slots.to(torch.int32).cpu())
    assert torch.equal(a.pool, b.pool)
    bt, n = torch.tensor([[1, 2]], dtype=torch.int32, device="cuda"), torch.tensor([150], dtype=torch.int32, device="cuda")
    ref = a.attend(q, bt, n)
    qt = q.transpose(1, 2).contiguous().transpose(1, 2)
    assert torch.equal(ref, a.attend(qt, bt.long().cpu(), n.long().cpu()))
    out, lse = a.attend(q, bt, n, return_lse=True)
    assert torch.equal(ref, out) and lse.shape == (1, 8)
    qc = q[:, None].expand(1, 3, 8, 128)
    ref = a.prefill_attend(qc.contiguous(), bt, n)
    assert torch.equal(ref, a.prefill_attend(qc, bt.long().cpu(), n.long().cpu()))


def test_wrong_arguments():
    import torch
    import turboquant_plus_b200 as tq
    cache, k, v, q = _cache(torch, tq)
    slots = torch.arange(150, device="cuda")
    with pytest.raises(AssertionError):
        cache.append(k, v[:, :1], slots)
    with pytest.raises(AssertionError):
        cache.append(k, v.float(), slots)
    with pytest.raises(ValueError):
        cache.append(k.cpu(), v.cpu(), slots)
    with pytest.raises(KeyError):
        cache.append(k.long(), v.long(), slots)
    with pytest.raises(AssertionError):
        cache.attend(q[..., :64], slots[None, :1], slots[:1])
    with pytest.raises(ValueError):                                  # 3 query heads over 2 KV heads
        cache.attend(q[:, :3], slots[None, :1], slots[:1])


@pytest.mark.parametrize("name", ["rotation", "centroids", "norm_correction", "S"])
def test_changed_constants(name):
    """Writing into an array that has been handed out, and assigning a new one, both reach the next call."""
    import torch
    import turboquant_plus_b200 as tq
    x = torch.randn((40, 64), device="cuda", dtype=torch.float64)
    t = tq.TurboQuant(64, 3, seed=1)
    holder = t.qjl if name == "S" else t.polar_quant
    before = t.dequantize(t.quantize(x))
    if name == "norm_correction":
        t.polar_quant.norm_correction = False
    else:
        getattr(holder, name)[...] *= -1.0 if name != "centroids" else 1.25     # in place
    changed = t.dequantize(t.quantize(x))
    assert not torch.allclose(before, changed) or name in ("rotation", "S")     # both signs of R (of S) code alike
    fresh = tq.TurboQuant(64, 3, seed=1, norm_correction=name != "norm_correction")
    if name != "norm_correction":
        setattr(fresh.qjl if name == "S" else fresh.polar_quant, name, np.array(getattr(holder, name)))
    code, want = t.quantize(x), fresh.quantize(x)
    assert torch.equal(code.mse_indices, want.mse_indices) and torch.equal(code.qjl_signs, want.qjl_signs)
    assert torch.allclose(t.dequantize(code), fresh.dequantize(want), rtol=1e-12, atol=1e-12)


def test_dropped_cache_is_freed_without_the_collector():
    """A cache with a captured step holds no reference cycle: its pool is gone when the last name is."""
    import torch
    from turboquant_plus_b200.layered import LayeredKVCache
    gc.collect()
    gc.disable()
    try:
        base = torch.cuda.memory_allocated()
        cache = LayeredKVCache(2, 128, 1, 2)
        cache.prepare_decode(1, 4, torch.zeros((1, 2), dtype=torch.int32), torch.zeros((1,), dtype=torch.int32))
        host = cache.host_buffers()
        cache.decode_step(*host)
        del cache, host
        assert torch.cuda.memory_allocated() <= base
    finally:
        gc.enable()
