"""tq_decode_attn_static accepts every shape whose partials fit its array under the coarsest plan, whatever plan a call with
a workspace of its own would take.  No buffers are passed: what is looked at is whether the size is refused."""
import ctypes as C

import pytest

from turboquant_plus_b200 import _native as nv

TOO_LARGE, STATIC = -5, 8 << 20
SLOTS = 2 * 148                                     # CTA places


def coarse_bytes(batch, hq, hkv, pages):
    """qrot, qproj, partials, their maxima and sums, tickets and status word."""
    items = batch * hkv
    chunk = min(pages, 32) if items >= SLOTS else -(-pages // -(-SLOTS // items))
    splits, rows = -(-pages // chunk), batch * hq
    up = lambda n: -(-n // 256) * 256
    return 2 * up(rows * 512) + up(rows * splits * 512) + up(rows * splits * 8) + 65536 * 4 + 256


@pytest.mark.parametrize("hkv,group", [(8, 8), (8, 4), (8, 1), (2, 8), (1, 4), (32, 1)])
def test_no_shape_is_lost_to_a_finer_plan(hkv, group):
    lib, layout = nv.load(), nv.CacheLayout()
    assert lib.tq_cache_layout_init(C.byref(layout), 128, 128, hkv, nv.FORMATS["q8_0"], nv.FORMATS["q8_0"]) == 0
    seen = 0
    for batch in (1, 2, 3, 5, 8, 12, 16, 20, 24, 31, 32, 36, 37, 64, 128, 300):
        for pages in (1, 2, 8, 33, 64, 256, 512, 1024):
            if coarse_bytes(batch, group * hkv, hkv, pages) > STATIC:
                continue
            seen += 1
            rc = lib.tq_decode_attn_static(None, None, C.byref(layout), None, None, pages, None, None, nv.F16, batch,
                                           group * hkv, 0.0, None, nv.F16, None)
            assert rc not in (0, TOO_LARGE), (batch, pages, lib.tq_last_error())
    assert seen > 40
