"""Decode attention over batches on both sides of the length at which the second split plan is taken: ragged, full and short
batches, one empty sequence, every form of the kernel, in stream order and after an append, against the same sequences
one at a time (a batch of one has one plan).

Tolerance: 2e-3 max-relative, that of the attention tests; the partials of another plan join in another order."""
import pytest

from tests.helpers import max_rel

pytestmark = pytest.mark.gpu
D = 128


@pytest.mark.parametrize("kf,vf,hkv,group,batch,pages,page_tokens", [
    ("turbo3", "turbo3", 8, 4, 16, 40, 128), ("turbo3", "turbo3", 8, 4, 24, 40, 128), ("turbo2", "turbo3", 2, 8, 64, 40, 128),
    ("turbo4", "turbo4", 8, 4, 20, 40, 128), ("prod3", "turbo3", 8, 2, 24, 24, 128), ("prod4", "turbo4", 4, 8, 40, 24, 128),
    ("q8_0", "turbo2", 8, 4, 12, 40, 128), ("turbo3", "turbo3", 8, 4, 16, 40, 64), ("turbo3", "turbo3", 1, 4, 290, 9, 128)])
def test_ragged_batches(kf, vf, hkv, group, batch, pages, page_tokens):
    import torch
    import turboquant_plus_b200 as tq
    gen = torch.Generator(device="cuda").manual_seed(batch)
    ctx = pages * page_tokens
    cache = tq.PagedKVCache(D, hkv, batch * pages, page_tokens, kf, vf, seed=42)
    for lo in range(0, batch * ctx, 16384):
        n = min(16384, batch * ctx - lo)
        k, v = (torch.randn((n, hkv, D), device="cuda", generator=gen).half() for _ in range(2))
        cache.append(k, v, torch.arange(lo, lo + n, device="cuda"))
    bt = torch.randperm(batch * pages, device="cuda", generator=gen).to(torch.int32).view(batch, pages)
    q = torch.randn((batch, hkv * group, D), device="cuda", generator=gen).half()
    even = torch.linspace(ctx // 32, ctx, batch).round().to(torch.int32)
    ragged = even[torch.randperm(batch, generator=torch.Generator().manual_seed(1))]
    ragged[3] = 0
    one_long = torch.full((batch,), 5, dtype=torch.int32)
    one_long[1] = ctx
    for lens in (ragged, torch.full((batch,), ctx), torch.full((batch,), 9 * ctx // 10), torch.full((batch,), 1), one_long):
        sl = lens.to(torch.int32).cuda()
        ones = [cache.attend(q[b:b + 1], bt[b:b + 1], sl[b:b + 1], return_lse=True) for b in range(batch)]
        want, lse_want = (torch.cat(t) for t in zip(*ones))
        live = lens > 0
        for overlap in (False, "append"):
            out, lse = cache.attend(q, bt, sl, overlap=overlap, return_lse=True)
            assert cache.kernel_status() == 0 and torch.equal(out, cache.attend(q, bt, sl, overlap=overlap))
            assert max_rel(out[live].cpu().numpy(), want[live].cpu().numpy()) < 2e-3
            assert torch.allclose(lse[live], lse_want[live], atol=1e-3) and not out[~live].any()
