"""Appends on both sides of the size at which the two-tensor kernel lets its successor come up late, one after the other into
the same slots and followed by the attention call that reads them: the records of each append and the outputs are those
of the same calls with a synchronisation between them."""
import pytest

pytestmark = pytest.mark.gpu
D = 128


@pytest.mark.parametrize("fmt", ["turbo2", "turbo3", "turbo4"])
@pytest.mark.parametrize("tokens", [1, 1183, 1184, 1185, 4096])     # 8 heads: 296 CTAs of 64 vectors for the two tensors at 1,184
def test_chained_appends(fmt, tokens):
    import torch
    import turboquant_plus_b200 as tq
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    n_pages = -(-tokens // 128)
    rows = [torch.randn(tokens, 8, D, device="cuda", generator=gen).half() for _ in range(4)]
    q = torch.randn(1, 32, D, device="cuda", generator=gen).half()
    table = torch.arange(n_pages, device="cuda", dtype=torch.int32).view(1, -1)
    lens = torch.tensor([tokens], device="cuda", dtype=torch.int32)
    slots = torch.arange(tokens, device="cuda")
    got = []
    for sync in (True, False):
        cache = tq.PagedKVCache(D, 8, n_pages, 128, fmt, fmt, seed=42)
        cache.pool.zero_()
        ws = cache.workspace(1, 32, n_pages)
        torch.cuda.synchronize()
        outs = []
        for k, v in ((rows[0], rows[1]), (rows[2], rows[3])):
            cache.append(k, v, slots)
            if sync:
                torch.cuda.synchronize()
            outs.append(cache.attend(q, table, lens, workspace=ws))
            if sync:
                torch.cuda.synchronize()
        cache.append(rows[0], rows[1], slots)
        cache.append(rows[2], rows[3], slots)
        torch.cuda.synchronize()
        got.append((outs, cache.pool.clone()))
    assert all(torch.equal(a, b) for a, b in zip(got[0][0], got[1][0])) and torch.equal(got[0][1], got[1][1])
