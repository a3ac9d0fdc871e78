"""Chains of attention calls on both sides of the sizes at which the form of the kernel changes (pages per CTA, splits, heads,
4-bit tables), against the same calls one by one in stream order.

Tolerance: 2e-3 max-relative, that of the attention tests; the forms join their partial sums in different orders."""
import pytest

from tests.helpers import max_rel

pytestmark = pytest.mark.gpu
D = 128


@pytest.mark.parametrize("kf,vf", [("turbo3", "turbo3"), ("turbo4", "turbo4"), ("turbo4", "turbo3"), ("turbo3", "turbo4"),
                                   ("q8_0", "turbo4"), ("q8_0", "turbo2"), ("prod4", "turbo4")])
@pytest.mark.parametrize("hkv,group,batch,ctx", [(8, 4, 32, 100), (8, 4, 16, 300), (8, 4, 16, 700), (1, 4, 1, 4000),
                                                 (8, 8, 32, 250), (8, 8, 4, 3000), (8, 6, 1, 4000), (2, 8, 1, 9000), (8, 5, 1, 40000)])
def test_chain_of_every_form(kf, vf, hkv, group, batch, ctx):
    import torch
    import turboquant_plus_b200 as tq
    gen = torch.Generator(device="cuda").manual_seed(ctx)
    pages = -(-ctx // 128)
    cache = tq.PagedKVCache(D, hkv, batch * pages, 128, kf, vf, seed=42)
    for lo in range(0, batch * pages * 128, 16384):
        n = min(16384, batch * pages * 128 - lo)
        k, v = (torch.randn((n, hkv, D), device="cuda", generator=gen).half() for _ in range(2))
        cache.append(k, v, torch.arange(lo, lo + n, device="cuda"))
    bt = torch.randperm(batch * pages, device="cuda", generator=gen).to(torch.int32).view(batch, pages)
    sl = torch.full((batch,), ctx, dtype=torch.int32, device="cuda")
    qs = [torch.randn((batch, hkv * group, D), device="cuda", generator=gen).half() for _ in range(3)]
    want = [cache.attend(q, bt, sl) for q in qs]
    torch.cuda.synchronize()
    for _ in range(2):
        got = [cache.attend(q, bt, sl, overlap="q" if i else False, chain_head=not i) for i, q in enumerate(qs)]
        torch.cuda.synchronize()
        assert cache.kernel_status() == 0
        for a, b in zip(got, want):
            assert max_rel(a.float().cpu().numpy(), b.float().cpu().numpy()) < 2e-3
