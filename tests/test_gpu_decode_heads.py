"""Decode attention for every group size of the two specialised forms (1..4 and 5..8 query heads per KV head) and every
format pair, in stream order, in a chain and after an append, against dequantize-then-attend.

Tolerance: 2e-3 max-relative, that of the attention tests, against the rows that the cache holds (an oracle that quantizes
the inputs itself takes a neighbouring index at one coordinate in some 10^5, up to 3e-2 of an output row)."""
import numpy as np
import pytest

from oracle import tq_oracle as o
from tests.helpers import D, fill_cache, max_rel, stored_rows
from tests.test_gpu_attention import TOL

pytestmark = pytest.mark.gpu

PAIRS = [("turbo2", "turbo2"), ("turbo2", "turbo4"), ("turbo3", "turbo3"), ("turbo3", "turbo4"), ("turbo4", "turbo2"),
         ("turbo4", "turbo3"), ("turbo4", "turbo4"), ("q8_0", "turbo2"), ("q8_0", "turbo4"), ("q8_0", "q8_0"),
         ("prod2", "turbo3"), ("prod3", "turbo2"), ("prod3", "turbo4"), ("prod4", "turbo3"), ("prod4", "turbo4")]


@pytest.mark.parametrize("kf,vf", PAIRS)
@pytest.mark.parametrize("group", [3, 4, 5, 6, 7, 8])
def test_decode_heads(kf, vf, group):
    import torch
    import turboquant_plus_b200 as tq
    rng = np.random.default_rng(group)
    hkv, lens = 2, [1, 16, 127, 128, 129, 1100]
    cache = tq.PagedKVCache(D, hkv, num_pages=16, k_format=kf, v_format=vf, seed=42)
    ks = [rng.standard_normal((n, hkv, D)).astype(np.float32) * 3 for n in lens]
    vs = [rng.standard_normal((n, hkv, D)).astype(np.float32) for n in lens]
    bt = fill_cache(cache, ks, vs, lens, rng).cuda()
    sl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    q = rng.standard_normal((len(lens), hkv * group, D)).astype(np.float32)
    qt = torch.as_tensor(q).cuda()
    want = []
    for b, n in enumerate(lens):
        pages = bt[b, :-(-n // 128)].cpu().numpy()
        kh, vh = (stored_rows(cache, w, pages, n).transpose(1, 0, 2)[None] for w in "kv")
        want.append(o.attend_gqa(q[b:b + 1].astype(np.float64), kh, vh, [n])[0])
    for mode in (False, True, "q", "append"):
        out, lse = cache.attend(qt, bt, sl, overlap=mode, return_lse=True)
        again = cache.attend(qt, bt, sl, overlap=mode)
        assert cache.kernel_status() == 0 and torch.equal(out, again) and torch.isfinite(lse).all()
        err = max(max_rel(out[b].cpu().numpy().reshape(-1, D), want[b].reshape(-1, D)) for b in range(len(lens)))
        assert err < TOL, f"{kf}/{vf} {group} heads, overlap={mode}: {err}"
