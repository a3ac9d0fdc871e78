"""Decode attention for every group size of the two specialised forms (1..4 and 5..8 query heads per KV head) and every
format pair, in stream order, in a chain and after an append, against dequantize-then-attend.

Tolerance: 2e-3 max-relative, that of the attention tests, for the arithmetic of the kernels.  The oracle quantizes the
inputs itself: a coordinate within rounding of a decision boundary may take the neighbouring index there (1 in some 10^5).
In a value that moves one rotated coordinate by a level step, at most 0.81 ||v|| / sqrt(d) = 0.81 (3 bits, outermost;
||v|| ~ sqrt(d)), i.e. every output coordinate by 0.81 / sqrt(d) = 0.072 times the token's weight, against a row maximum of
about 2.5: up to 3e-2 where one of few tokens has all the weight.  One sequence per case may show that."""
import numpy as np
import pytest

from tests.helpers import D, fill_cache, max_rel
from tests.test_gpu_attention import TOL, oracle_attention

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
    want = oracle_attention(cache, ks, vs, q, lens)
    for mode in (False, True, "q", "append"):
        out, lse = cache.attend(qt, bt, sl, overlap=mode, return_lse=True)
        again = cache.attend(qt, bt, sl, overlap=mode)
        assert cache.kernel_status() == 0 and torch.equal(out, again) and torch.isfinite(lse).all()
        err = sorted(max_rel(out[b].cpu().numpy().reshape(-1, D), want[b].reshape(-1, D)) for b in range(len(lens)))
        assert err[-2] < TOL and err[-1] < 3e-2, f"{kf}/{vf} {group} heads, overlap={mode}: {err}"
