"""A decode step whose rows come and go in parts: layer counts and batches on both sides of the rule, format groups that
lie together, at the ends and interleaved, against the same step through pageable buffers (one copy, one part)."""
import pytest

pytestmark = pytest.mark.gpu
D = 128


@pytest.mark.parametrize("L,B,hq,hkv,dtype", [(6, 16, 32, 8, "float16"), (5, 16, 32, 8, "float16"), (1, 96, 32, 8, "float16"),
                                               (33, 8, 64, 8, "bfloat16"), (17, 3, 16, 2, "float16")])
@pytest.mark.parametrize("table", ["one", "ends", "mixed"])
def test_step_in_parts(L, B, hq, hkv, dtype, table):
    import torch
    from turboquant_plus_b200.layered import LayeredKVCache, boundary_format_table
    dt = getattr(torch, dtype)
    formats = {"one": [("turbo3", "turbo3")] * L, "ends": boundary_format_table(L, keep=min(2, (L - 1) // 2)),
               "mixed": [(("turbo3", "turbo3"), ("turbo4", "turbo2"))[i % 2] for i in range(L)]}[table]
    lens = torch.tensor([3 + 17 * b for b in range(B)], dtype=torch.int32)
    n_pages = 3 + 17 * B // 128
    gen = torch.Generator().manual_seed(L)
    bt = torch.arange(B * n_pages, dtype=torch.int32).view(B, n_pages)
    outs = []
    for pinned in (False, True):
        cache = LayeredKVCache(L, D, hkv, B * n_pages, formats=formats, seed=42)
        for whole, members in cache.groups:
            whole.pool.zero_()
        cache.prepare_decode(B, hq, bt, lens, dtype=dt)
        gen.manual_seed(L)
        got = []
        for step in range(2):
            host = cache.host_buffers() if pinned else tuple(torch.zeros(s, dtype=dt) for s in
                                                             ((L, B, hq, D), (L, B, hkv, D), (L, B, hkv, D), (L, B, hq, D)))
            for t in host[:3]:
                t.copy_(torch.randn(t.shape, generator=gen).to(dt))
            for _ in range(2):
                got.append(cache.decode_step(*host).clone())
        assert torch.equal(cache._step["len"].cpu(), lens + 4)
        outs.append((got, [whole.pool.clone() for whole, _ in cache.groups]))
    for a, b in zip(outs[0][1], outs[1][1]):
        assert torch.equal(a, b)                    # the appended records
    for a, b in zip(outs[0][0], outs[1][0]):
        # the first call of a part reads its queries after the wait, in the same order of operations
        assert torch.equal(a, b)
