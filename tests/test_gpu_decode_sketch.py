"""The sign sketch's share of a score, as sums over its set bits: projected queries of any magnitude, a zero head, tile remainders.
Against fp64 over the stored rows: outputs, and the share alone, as half of the difference that the inverted sketch makes to a
score.  Bound of the outputs, of the largest output row's length: fp16 probabilities and fp16 values each round by
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


@pytest.mark.parametrize("factor", [2.0 ** -6, 1.0, 2.0 ** 6])
@pytest.mark.parametrize("group", [1, 4, 7])
@pytest.mark.parametrize("fmt", ["prod2", "prod3", "prod4"])
def test_sketch_share(fmt, group, factor):
    """Sequences of one token: the log-sum-exp is the score.  Bound: the projected query's elements are off by 2^-20 in all (seven
    stages of butterflies, hi and lo halves), a sum of 128 terms by as much again, each score and its way to the log-sum-exp by
    eight roundings of 2^-24.  (With the lo halves lost the share would be off by 2^-9 of the projected query's length.)"""
    import torch
    import turboquant_plus_b200 as tq
    from perf.cases import _records
    n, hq = 40, HKV * group
    gen = torch.Generator(device="cuda").manual_seed(group)
    cache = tq.PagedKVCache(D, HKV, 2 * n, 128, fmt, "turbo3", seed=42)
    cache.pool.zero_()
    k, v = (torch.randn(n, HKV, D, device="cuda", generator=gen).half() for _ in range(2))
    cache.append(k, v, 128 * torch.arange(n, device="cuda"))
    cache.pool[n:] = cache.pool[:n]
    _records(cache)["k_sketch"][n:] ^= 0xFF
    q = torch.randn(n, hq, D, device="cuda", generator=gen)
    q[:, 0, 0] = 10.0
    q[0, hq - 1] = 0.0
    table = torch.arange(2 * n, device="cuda", dtype=torch.int32).view(-1, 1)
    lens = torch.ones(2 * n, device="cuda", dtype=torch.int32)
    scale = 1.0 / np.sqrt(D)
    _, lse = cache.attend(torch.cat([q, q]) * factor, table, lens, scale=scale / factor, return_lse=True)
    lse = lse.double().cpu().numpy()
    keys = stored_rows(cache, "k", list(range(2 * n)), 2 * n * 128)[::128].repeat(group, axis=1)
    part = (keys[:n] - keys[n:]) / 2
    q = q.double().cpu().numpy()
    share = (q * part).sum(2) * scale
    mass = np.abs(q @ cache.k_quantizer.qjl.S.T).sum(2) * np.linalg.norm(part, axis=2) / np.sqrt(D) * scale
    bound = 2.0 ** -19 * mass + 2.0 ** -21 * np.abs(lse).reshape(2, n, hq).max(0)
    err = np.abs((lse[:n] - lse[n:]) / 2 - share)
    assert (err <= bound).all(), (err / np.maximum(bound, 1e-300)).max()


@pytest.mark.parametrize("group", [1, 4, 7])
def test_tiny_queries(group):
    """Queries down to the smallest numbers of their type: scores of next to nothing, the outputs are those of zero queries."""
    import torch
    import turboquant_plus_b200 as tq
    n, hq = 300, HKV * group
    gen = torch.Generator(device="cuda").manual_seed(group)
    cache = tq.PagedKVCache(D, HKV, 3, 128, "prod3", "turbo3", seed=42)
    k, v = (torch.randn(n, HKV, D, device="cuda", generator=gen).half() for _ in range(2))
    cache.append(k, v, torch.arange(n, device="cuda"))
    powers = torch.arange(20, 46, device="cuda")
    q = torch.randn(len(powers), hq, D, device="cuda", generator=gen) * (10.0 ** -powers.double())[:, None, None].float()
    table = torch.arange(3, device="cuda", dtype=torch.int32).repeat(len(powers), 1)
    lens = torch.full((len(powers),), n, device="cuda", dtype=torch.int32)
    out, zero = cache.attend(q, table, lens), cache.attend(torch.zeros_like(q), table, lens)
    assert torch.equal(out, zero) and bool(out.isfinite().all())
