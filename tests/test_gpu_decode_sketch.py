"""The sign sketch's share of a score, as sums over its set bits: projected queries of any magnitude, a zero head, tile remainders.
Against fp64 over the stored rows.  Bound, of the largest output row's length: fp16 probabilities and fp16 values each round by
2^-11 (2^-10 together); keys rounded to fp16 add at most 2^-11 of the largest score twice (a weight and the denominator)."""
import numpy as np
import pytest

from tests.helpers import stored_rows

pytestmark = pytest.mark.gpu
D, HKV = 128, 2


@pytest.mark.parametrize("factor", [2.0 ** -6, 1.0, 2.0 ** 6])
@pytest.mark.parametrize("group", [1, 4, 7])
@pytest.mark.parametrize("fmt", ["prod2", "prod3", "prod4"])
def test_sketch_scores(fmt, group, factor):
    import torch
    import turboquant_plus_b200 as tq
    n, hq = 1003, HKV * group
    gen = torch.Generator(device="cuda").manual_seed(group)
    pages = -(-n // 128)
    cache = tq.PagedKVCache(D, HKV, pages, 128, fmt, "turbo3", seed=42)
    k, v = (torch.randn(n, HKV, D, device="cuda", generator=gen).half() for _ in range(2))
    cache.append(k, v, torch.arange(n, device="cuda"))
    q = torch.randn(1, hq, D, device="cuda", generator=gen)
    q[0, 0, 0] = 10.0
    q[0, hq - 1] = 0.0
    table = torch.arange(pages, device="cuda", dtype=torch.int32).view(1, -1)
    lens = torch.tensor([n], device="cuda", dtype=torch.int32)
    scale = 1.0 / np.sqrt(D)
    out = cache.attend(q * factor, table, lens, scale=scale / factor)[0].double().cpu().numpy()
    keys, values = (stored_rows(cache, t, list(range(pages)), n).repeat(group, axis=1) for t in ("k", "v"))
    s = np.einsum("hd,nhd->hn", q[0].double().cpu().numpy(), keys) * scale
    p = np.exp(s - s.max(1, keepdims=True))
    ref = np.einsum("hn,nhd->hd", p / p.sum(1, keepdims=True), values)
    err = np.linalg.norm(out - ref, axis=1).max()
    assert err <= (2.0 ** -10 + 2 * np.abs(s).max() * 2.0 ** -11) * np.linalg.norm(ref, axis=1).max()
