"""Chunked prefill over q8_0 keys with elements beyond the fp16 range (bf16 and fp32 rows can hold them; the cache stores
int8 and a block scale), single CTAs and pairs, one and several splits, against dequantize-then-attend.

Tolerance: that of the attention tests.  The products int8 x scale of such a token are divided by 128 as operands; they
stay exact to 2^-32 of the token's largest element.  Queries are small in the large channel, so that the scores stay
moderate: multiples of 2^-24 after scaling, which fp16 holds."""
import numpy as np
import pytest

from oracle import tq_oracle as o
from tests.helpers import D, fill_cache, max_rel
from tests.test_gpu_attention import TOL, oracle_roundtrip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vf", ["turbo3", "q8_0"])
@pytest.mark.parametrize("group,chunk,lens", [(4, 16, [200, 33]), (4, 65, [4200, 300]), (8, 33, [700, 129])])
@pytest.mark.parametrize("largest", [1e5, 6e6])
def test_keys_beyond_fp16(vf, group, chunk, lens, largest):
    import torch
    import turboquant_plus_b200 as tq
    rng = np.random.default_rng(chunk)
    hkv, channel = 2, 77
    cache = tq.PagedKVCache(D, hkv, num_pages=sum(-(-n // 128) for n in lens) + 1, k_format="q8_0", v_format=vf, seed=42)
    ks = [rng.standard_normal((n, hkv, D)).astype(np.float32) for n in lens]
    vs = [rng.standard_normal((n, hkv, D)).astype(np.float32) for n in lens]
    for k in ks:                                                # every third token, both signs
        k[::3, :, channel] = largest * rng.uniform(-1, 1, k[::3].shape[:2])
    bt = fill_cache(cache, ks, vs, lens, rng)
    q = rng.standard_normal((len(lens), chunk, hkv * group, D)).astype(np.float32)
    q[..., channel] = np.round(q[..., channel] * 2**24 * 8 / largest) * 2.0**-20
    scale = 2.0**-4 / np.log2(np.e)                             # the kernel's scores are q k scale log2(e)
    out = cache.prefill_attend(torch.as_tensor(q).cuda(), bt, torch.tensor(lens), scale=scale).cpu().numpy()
    assert cache.kernel_status() == 0 and np.isfinite(out).all()
    for b, n in enumerate(lens):
        kh = np.stack([oracle_roundtrip(cache, ks[b][:, h], "k") for h in range(hkv)])[None]
        vh = np.stack([oracle_roundtrip(cache, vs[b][:, h], "v") for h in range(hkv)])[None]
        ref = o.attend_chunk_gqa(q[b:b + 1].astype(np.float64) * (scale * np.sqrt(D)), kh, vh, [n])
        assert max_rel(out[b].reshape(-1, D), ref.reshape(-1, D)) < TOL
