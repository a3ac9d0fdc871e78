"""Decode calls whose splits are a cluster of CTAs merged in shared memory, and sequences that are one split, against attention over the
rows that the cache holds: one to eight splits, sequences shorter than others of their batch (whose later CTAs have nothing to do) and
empty ones, one to eight heads, the log-sum-exp, behind an append and in stream order.

Tolerance 2e-3 of the largest output of a row: fp16 operands of the products, 32-bit sums, as for the other decode forms."""
import numpy as np
import pytest

from oracle import tq_oracle as o
from tests.helpers import D, fill_cache, max_rel, stored_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,v", [("turbo3", "turbo3"), ("turbo4", "turbo2"), ("q8_0", "turbo2"), ("prod3", "turbo3")])
@pytest.mark.parametrize("group,lengths", [(4, [129]), (1, [1024]), (4, [1000, 3, 257]), (5, [700, 128, 1]), (8, [1024, 512]), (3, [640] * 4 + [385, 0]),
                                           (4, [128, 1, 77, 100])])
def test_splits_of_a_cluster(k, v, group, lengths):
    import torch
    import turboquant_plus_b200 as tq
    hkv = 2
    rng = np.random.default_rng(sum(lengths) + group)
    cache = tq.PagedKVCache(D, hkv, 60, 128, k, v, seed=42)
    kh, vh = ([rng.standard_normal((n, hkv, D)).astype(np.float16) for n in lengths] for _ in range(2))
    table = fill_cache(cache, kh, vh, lengths, rng)
    lens = torch.tensor(lengths, dtype=torch.int32)
    q = torch.as_tensor(rng.standard_normal((len(lengths), hkv * group, D)).astype(np.float16)).cuda()
    got = {}
    for overlap in (False, "append"):
        got[overlap], lse = cache.attend(q, table, lens, overlap=overlap, return_lse=True)
        assert cache.kernel_status() == 0
    assert torch.equal(got[False], got["append"])
    for b, n in enumerate(lengths):
        out = got[False][b].float().cpu().numpy()
        if n == 0:
            assert not out.any() and bool((lse[b] == -float("inf")).all())
            continue
        pages = table[b, :-(-n // 128)].tolist()
        rows = [stored_rows(cache, w, pages, n).transpose(1, 0, 2)[None] for w in "kv"]
        qb = q[b:b + 1].double().cpu().numpy()
        assert max_rel(out, o.attend_gqa(qb, *rows, [n])[0]) < 2e-3
        scores = np.einsum("hd,htd->ht", qb[0], np.repeat(rows[0][0], group, axis=0)) / np.sqrt(D)
        want = scores.max(1) + np.log(np.exp(scores - scores.max(1, keepdims=True)).sum(1))
        assert np.abs(lse[b].cpu().numpy() - want).max() < 2e-3


@pytest.mark.parametrize("dtype", ["float16", "bfloat16", "float32"])
@pytest.mark.parametrize("lengths", [[517], [100], [1000, 257, 40]])
def test_captured_with_its_append(lengths, dtype):
    """The new token's append and the attention behind it as a graph, in every type of result: bit for bit what the calls give one by one,
    and within one rounding of the type of the fp32 results."""
    import torch
    import turboquant_plus_b200 as tq
    hkv, group = 2, 4
    rng = np.random.default_rng(sum(lengths))
    cache = tq.PagedKVCache(D, hkv, 60, 128, "turbo3", "turbo3", seed=42)
    kh, vh = ([rng.standard_normal((n, hkv, D)).astype(np.float16) for n in lengths] for _ in range(2))
    table = fill_cache(cache, kh, vh, lengths, rng)
    pages, lens = torch.as_tensor(table).to(device="cuda", dtype=torch.int32), torch.tensor(lengths, dtype=torch.int32, device="cuda")
    last = lens.long() - 1
    slots = pages.long()[torch.arange(len(lengths), device="cuda"), last // 128] * 128 + last % 128
    k, v = (torch.as_tensor(rng.standard_normal((len(lengths), hkv, D)).astype(np.float16)).cuda() for _ in range(2))
    q = torch.as_tensor(rng.standard_normal((len(lengths), hkv * group, D)).astype(np.float16)).cuda().to(getattr(torch, dtype))
    ws = cache.workspace(len(lengths), hkv * group, pages.shape[1])

    def step(out):
        cache.append(k, v, slots)
        cache.attend(q, pages, lens, out=out, workspace=ws, overlap="append")

    eager, captured, graph = torch.empty_like(q), torch.zeros_like(q), torch.cuda.CUDAGraph()
    step(eager)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        step(captured)
    for _ in range(3):
        captured.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(captured, eager) and cache.kernel_status(ws) == 0
    graph.reset()
    exact = cache.attend(q.float(), pages, lens)
    eps = {"float16": 2.0 ** -11, "bfloat16": 2.0 ** -8, "float32": 2.0 ** -20}[dtype]
    assert bool(((eager.float() - exact.float()).abs() <= eps * exact.float().abs() + 1e-7).all())
