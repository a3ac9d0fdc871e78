"""Bounded waits of the tensor-core quantize and dequantize kernels that run out: a call whose first CTA never reports one product of
its second tile, or third, as done.  What it did compute is right, the rest is marked as not a number, the status word says so once, and
the same calls then run as before.  And a call one of whose roles is late, which gives up nothing."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu
D, TILE = 128, 128


def _status(nv):
    import torch
    torch.cuda.synchronize()
    word = ctypes.c_int32()
    nv.call("tq_quantize_status_sync", ctypes.byref(word))
    return word.value


def _first_cta(n, sms):
    """Tile of every vector, counted within its CTA, where that is the first one; else -1."""
    import torch
    tile = torch.arange(n, device="cuda") // TILE
    return torch.where(tile % sms == 0, tile // sms, -1)


def _check(seen, right, at, tile=1):
    """Rows of the outputs in `seen`, the first of which marks what was given up: other CTAs and tiles before `tile` are right, `tile`
    is not there."""
    import torch
    lost = seen[0].reshape(len(at), -1).isnan().any(1)
    assert bool(lost[at == tile].all()) and not bool(lost[at < tile - 1].any())
    assert tile > 1 or not bool(lost[at < tile].any())
    for a, b in zip(seen, right):
        a, b = a.reshape(len(at), -1), b.reshape(len(at), -1)
        assert torch.equal(a[~lost], b[~lost])
        assert not a.is_floating_point() or bool(a[lost].isnan().all())


def test_long_append_gives_up():
    import torch
    import turboquant_plus_b200 as tq
    from turboquant_plus_b200 import _native as nv
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = TILE * 15 * sms + 37                                  # 15 or 16 tiles a CTA: more than the rings hold
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, D, device="cuda", generator=gen).half()
    q = tq.PolarQuant(D, 3, seed=1, rotation="wht")
    right = q.quantize_device(x, packed=True, want_scale=True)
    right = right["norm"], right["scale"], right["packed"]
    assert _status(nv) == 0
    seen = torch.zeros_like(right[0]), torch.zeros_like(right[1]), torch.zeros_like(right[2])
    nv.call("tq_selftest_quantize_gives_up", q._native(x.device).handle, nv.ptr(x), D, n, nv.ptr(seen[2]), nv.ptr(seen[0]),
            nv.ptr(seen[1]), None, None, nv.stream_ptr())
    assert _status(nv) == 1 and _status(nv) == 0
    _check(seen, right, _first_cta(n, sms))
    again = q.quantize_device(x, packed=True, want_scale=True)
    assert torch.equal(again["packed"], right[2]) and torch.equal(again["scale"], right[1]) and _status(nv) == 0


def test_dense_calls_give_up():
    import torch
    import turboquant_plus_b200 as tq
    from turboquant_plus_b200 import _native as nv
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = TILE * 3 * sms + 37
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, D, device="cuda", generator=gen)
    q = tq.TurboQuant(D, 3, seed=1)
    out = q.quantize_device(x)
    right = out["norm"], out["rnorm"], out["idx"], out["qjl"]
    seen = tuple(torch.zeros_like(t) for t in right)
    handle, at = q._native(x.device).handle, _first_cta(n, sms)
    nv.call("tq_selftest_quantize_gives_up", handle, nv.ptr(x), D, n, nv.ptr(seen[2]), nv.ptr(seen[0]), None, nv.ptr(seen[3]),
            nv.ptr(seen[1]), nv.stream_ptr())
    assert _status(nv) == 1 and _status(nv) == 0
    _check(seen, right, at)

    def back():
        y = torch.empty(n, D, device="cuda", dtype=torch.float64)
        nv.call("tq_dequantize", handle, None, nv.ptr(right[2]), nv.ptr(right[0]), nv.ptr(right[3]), nv.ptr(right[1]), 1.0, n, nv.ptr(y),
                nv.F64, nv.stream_ptr())
        return y

    y, lost = back(), torch.zeros(n, D, device="cuda", dtype=torch.float64)
    nv.call("tq_selftest_dequantize_gives_up", handle, nv.ptr(right[2]), nv.ptr(right[0]), nv.ptr(right[3]), nv.ptr(right[1]), n,
            nv.ptr(lost), nv.stream_ptr())
    assert _status(nv) == 1 and _status(nv) == 0
    _check((lost,), (y,), at)
    assert bool(lost[at >= 1].isnan().all())
    again = q.quantize_device(x)
    assert torch.equal(again["idx"], right[2]) and torch.equal(again["qjl"], right[3]) and torch.equal(back(), y) and _status(nv) == 0


@pytest.mark.parametrize("tiles", [3, 4, 5])
def test_dense_call_without_a_sketch_gives_up(tiles):
    """In the last tile of a CTA, in the last but one and earlier: the rows look at a tile's sums a tile later."""
    import torch
    import turboquant_plus_b200 as tq
    from turboquant_plus_b200 import _native as nv
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = TILE * (tiles - 1) * sms + 37
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, D, device="cuda", generator=gen)
    q = tq.TurboQuantMSE(D, 2, seed=1).polar_quant
    out = q.quantize_device(x)
    right = out["norm"], out["idx"]
    seen = tuple(torch.zeros_like(t) for t in right)
    nv.call("tq_selftest_quantize_gives_up", q._native(x.device).handle, nv.ptr(x), D, n, nv.ptr(seen[1]), nv.ptr(seen[0]), None, None,
            None, nv.stream_ptr())
    assert _status(nv) == 1 and _status(nv) == 0
    at = _first_cta(n, sms)
    _check(seen, right, at, 2)
    assert bool(seen[0][at >= 2].isnan().all())
    again = q.quantize_device(x)
    assert torch.equal(again["idx"], right[1]) and _status(nv) == 0


@pytest.mark.parametrize("tiles", [1, 2, 5])
def test_outputs_that_nobody_decides(tiles):
    """The warp that decides outputs close to a boundary leaves at once: the call says so, and what it marks as computed is right."""
    import torch
    import turboquant_plus_b200 as tq
    from tests.test_gpu_dense_digits import _next_to_boundaries
    from turboquant_plus_b200 import _native as nv
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = TILE * (tiles - 1) * sms + 37
    q = tq.TurboQuantMSE(D, 2, seed=1).polar_quant
    x = _next_to_boundaries(q, n, n)
    right = q.quantize_device(x)
    idx, norm = torch.zeros_like(right["idx"]), torch.zeros_like(right["norm"])
    nv.call("tq_selftest_quantize_role", q._native(x.device).handle, nv.ptr(x), D, n, nv.ptr(idx), nv.ptr(norm), 1, nv.stream_ptr())
    assert _status(nv) == 1 and _status(nv) == 0
    lost = norm.isnan()
    assert bool(lost.any()) and torch.equal(idx[~lost], right["idx"][~lost]) and torch.equal(norm[~lost], right["norm"][~lost])


@pytest.mark.parametrize("tiles", [1, 2, 5])
def test_products_that_come_late(tiles):
    """The warp that issues the products comes late to every operand, when the rows have already written the next one."""
    import torch
    import turboquant_plus_b200 as tq
    from turboquant_plus_b200 import _native as nv
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = TILE * (tiles - 1) * sms + 37
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, D, device="cuda", generator=gen)
    q = tq.TurboQuantMSE(D, 2, seed=1).polar_quant
    right = q.quantize_device(x)
    idx, norm = torch.zeros_like(right["idx"]), torch.zeros_like(right["norm"])
    nv.call("tq_selftest_quantize_role", q._native(x.device).handle, nv.ptr(x), D, n, nv.ptr(idx), nv.ptr(norm), 0, nv.stream_ptr())
    assert _status(nv) == 0
    assert torch.equal(idx, right["idx"]) and torch.equal(norm, right["norm"])
