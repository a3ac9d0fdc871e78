"""Long appends, which take 128 vectors a tensor-core tile, against the same rows appended in short pieces, which the warp-level
kernel takes: vectors around a tile's edge, head counts that leave a ragged last tile, zero rows, tokens without a slot.
Both form every sum behind an index in the same order: indices are equal.  Scales come from sums of counts in another order:
six roundings of 2^-24 in all.  PROD keys take the warp-level kernel at every length: all of their record is equal."""
import pytest

pytestmark = pytest.mark.gpu
D = 128


def _fields(cache):
    import torch
    from perf.cases import _records
    out = {}
    for name, view in _records(cache).items():
        out[name] = view.reshape(cache.num_pages, cache.num_kv_heads, 128, -1)
    return out


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("k,v,vectors", [("turbo2", "turbo2", 24568), ("turbo3", "turbo3", 24567), ("turbo3", "turbo3", 24568),
                                         ("turbo4", "turbo4", 24569), ("turbo3", "turbo3", 24703), ("turbo3", "turbo3", 75777),
                                         ("turbo4", "turbo4", 131072), ("q8_0", "turbo2", 262849), ("prod3", "turbo3", 284673)])
def test_long_append_equals_short_ones(k, v, vectors, dtype):
    import torch
    import turboquant_plus_b200 as tq
    heads = 3 if vectors % 3 == 0 else 1
    tokens = vectors // heads
    gen = torch.Generator(device="cuda").manual_seed(vectors)
    rows = []
    for _ in range(2):
        x = torch.randn(tokens, heads, D, device="cuda", generator=gen)
        x *= torch.exp(0.5 * torch.randn(tokens, heads, 1, device="cuda", generator=gen))
        x[5] = 0
        x[tokens - 1, heads - 1] = 0
        rows.append(x.to(getattr(torch, dtype)))
    n_pages = -(-tokens // 128)
    slots = torch.randperm(n_pages, generator=gen, device="cuda")[torch.arange(tokens, device="cuda") // 128] * 128 \
        + torch.arange(tokens, device="cuda") % 128
    slots[7] = -1
    got = []
    for piece in (tokens, 1000):
        cache = tq.PagedKVCache(D, heads, n_pages, 128, k, v, seed=42)
        cache.pool.fill_(0xA5)
        for lo in range(0, tokens, piece):
            cache.append(rows[0][lo:lo + piece], rows[1][lo:lo + piece], slots[lo:lo + piece])
        got.append(cache)
    a, b = (_fields(c) for c in got)
    for t, fmt in (("k", k), ("v", v)):
        assert torch.equal(a[t], b[t])
        if fmt == "q8_0" or fmt.startswith("prod"):
            for name in a:
                assert not name.startswith(t) or torch.equal(a[name], b[name])
            continue
        written = torch.zeros(n_pages * 128, heads, device="cuda", dtype=torch.bool)
        written[slots[slots >= 0]] = True
        written = written.view(n_pages, 128, heads).transpose(1, 2)
        sa, sb = a[t + "_scale"][..., 0][written], b[t + "_scale"][..., 0][written]
        assert bool(((sa - sb).abs() <= 6 * 2.0 ** -24 * sb.abs()).all())
