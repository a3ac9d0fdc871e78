"""Chunked prefill over q8_0 and PROD tensors on the tcgen05 kernel, against dequantize-then-attend on the visible prefix.

Tolerance: 2e-3 max-relative, that of the attention tests.  The K operands of these formats are exact (hi + lo fp16
terms), so what is left is the rounding of P, of the fp16 V operand and of the fp16 centroid table, 2^-12 each."""
import numpy as np
import pytest

from oracle import tq_oracle as o
from tests.helpers import D, fill_cache, max_rel
from tests.test_gpu_attention import TOL, oracle_roundtrip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kf,vf,mode,group,chunk", [
    ("q8_0", "turbo2", "wht", 4, 24), ("q8_0", "turbo3", "wht", 8, 17), ("q8_0", "turbo4", "wht", 1, 128),
    ("q8_0", "q8_0", "wht", 4, 33), ("prod2", "turbo2", "wht", 4, 24), ("prod2", "turbo3", "wht", 2, 9),
    ("prod3", "turbo2", "wht", 8, 16), ("prod3", "turbo3", "wht", 4, 40), ("prod3", "turbo4", "wht", 1, 129),
    ("prod4", "turbo3", "wht", 4, 24), ("prod4", "turbo4", "wht", 8, 1), ("prod3", "turbo3", "dense", 4, 24)])
def test_prefill_formats(kf, vf, mode, group, chunk):
    """Lengths at page edges, a chunk longer than its sequence (its first queries see nothing), a split page range."""
    import torch
    import turboquant_plus_b200 as tq
    rng = np.random.default_rng(37)
    hkv = 2
    lens = [max(chunk - 3, 1), 128, 129, 257, 2305]
    cache = tq.PagedKVCache(D, hkv, num_pages=28, k_format=kf, v_format=vf, seed=42, rotation=mode)
    ks = [np.stack([o.rope_rotate(o.synth_keys(n, seed=9 * b + h), np.arange(n)) for h in range(hkv)], axis=1)
          for b, n in enumerate(lens)]
    vs = [rng.standard_normal((n, hkv, D)).astype(np.float32) for n in lens]
    bt = fill_cache(cache, ks, vs, lens, rng)
    q = rng.standard_normal((len(lens), chunk, hkv * group, D)).astype(np.float32)
    qt = torch.as_tensor(q).cuda()
    out = cache.prefill_attend(qt, bt, torch.tensor(lens)).cpu().numpy()
    assert cache.kernel_status() == 0
    assert np.array_equal(out, cache.prefill_attend(qt, bt, torch.tensor(lens)).cpu().numpy())
    for b, n in enumerate(lens):
        lo = max(0, chunk - n)                                # queries before the sequence's start: zeros
        assert not out[b, :lo].any()
        kh = np.stack([oracle_roundtrip(cache, ks[b][:, h], "k") for h in range(hkv)])[None]
        vh = np.stack([oracle_roundtrip(cache, vs[b][:, h], "v") for h in range(hkv)])[None]
        ref = o.attend_chunk_gqa(q[b:b + 1, lo:].astype(np.float64), kh, vh, [n])
        err = max_rel(out[b, lo:].reshape(-1, D), ref.reshape(-1, D))
        print(f"prefill {kf}/{vf} {mode} length {n}: max-rel {err:.2e}")
        assert err < TOL
    rows16 = cache.prefill_attend(qt.half(), bt, torch.tensor(lens))
    want16 = cache.prefill_attend(qt.half().float(), bt, torch.tensor(lens)).half()
    assert torch.equal(rows16, want16)
