"""Long appends, which take 128 vectors a tensor-core tile, against the same rows appended in short pieces, which the warp-level
kernel takes: vectors around a tile's edge, head counts that leave a ragged last tile, zero rows, tokens without a slot, rows of
exact zeros, of both ends of their type's range and beyond it, plain packed arrays.
Both form every sum behind an index in the same order: indices are equal.  Scales come from sums of counts in another order:
six roundings of 2^-24 in all.  PROD keys form all of their sums in the same order: all of their record is equal, bit for bit."""
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


# vectors per SM from which two tensors of one format, one beside another kernel, and PROD keys, take the tile kernel
PAIR, ALONE = 166, 1776
SKETCH = 332


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("k,v,heads,per_sm,more", [("turbo2", "turbo2", 1, PAIR, 0), ("turbo3", "turbo3", 1, PAIR, -1), ("turbo3", "turbo3", 3, PAIR, 2),
                                                   ("turbo4", "turbo4", 8, PAIR, 8), ("turbo3", "turbo3", 1, PAIR, 135), ("turbo3", "turbo3", 3, 512, 1),
                                                   ("turbo2", "turbo2", 8, 880, 8), ("turbo4", "turbo4", 3, 880, 2), ("q8_0", "turbo2", 8, ALONE, 8),
                                                   ("q8_0", "turbo4", 3, ALONE, 2), ("turbo3", "turbo3", 8, ALONE, 136), ("prod3", "turbo3", 3, 1923, 0),
                                                   ("prod3", "turbo3", 1, SKETCH, 0), ("prod3", "turbo2", 3, SKETCH, -1), ("prod4", "turbo4", 8, SKETCH, 136),
                                                   ("prod4", "turbo3", 3, 512, 1), ("prod3", "turbo3", 8, 1333, 8)])
def test_long_append_equals_short_ones(k, v, heads, per_sm, more, dtype):
    import torch
    import turboquant_plus_b200 as tq
    vectors = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
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


def _odd_rows(tokens, heads, dtype, gen):
    """Rows whose coordinates are exact zeros in number (few nonzeros of one magnitude, small integers, signed zeros), rows with
    outlier channels, and rows at the ends of the type's range or beyond it: row i is of kind i % 12."""
    import torch
    x = torch.randn(tokens * heads, D, device="cuda", generator=gen)
    i = torch.arange(tokens * heads, device="cuda")
    for kind, nonzeros in ((0, 1), (1, 2), (2, 4), (3, 8)):
        r = i[i % 12 == kind]
        at = torch.rand(len(r), D, device="cuda", generator=gen).argsort(1)[:, :nonzeros]
        sign = torch.randint(0, 2, at.shape, device="cuda", generator=gen) * 2.0 - 1.0
        x[r] = torch.zeros(len(r), D, device="cuda").scatter_(1, at, sign)
    r = i[i % 12 == 4]                                        # two equal neighbours
    at = torch.randint(0, D - 1, (len(r), 1), device="cuda", generator=gen)
    x[r] = torch.zeros(len(r), D, device="cuda").scatter_(1, torch.cat([at, at + 1], 1), 3.0)
    r = i[i % 12 == 5]
    x[r] = torch.randint(-7, 8, (len(r), D), device="cuda", generator=gen).float()
    r = i[i % 12 == 6]                                        # zeros of both signs
    x[r] = torch.where(torch.rand(len(r), D, device="cuda", generator=gen) < 0.9, torch.zeros_like(x[r]).copysign(x[r]), x[r].sign())
    x[i[i % 12 == 7], 3:7] *= 1000
    r = i[i % 12 == 8]                                        # channels of very different sizes
    x[r] *= torch.exp2(torch.randint(-8, 9, (len(r), D), device="cuda", generator=gen).float())
    big, small = (6e4, 6e-8) if dtype == "float16" else (3e38, 1e-38)
    r = i[i % 12 == 9]
    x[r] = torch.where((r % 2 == 0)[:, None], x[r].sign() * big, x[r] * small)
    r = i[i % 12 == 10]
    x[r, r % D] = torch.tensor([float("nan"), float("inf"), float("-inf")], device="cuda")[r % 36 // 12]
    return x.view(tokens, heads, D).to(getattr(torch, dtype))


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("norm_correction", [True, False])
@pytest.mark.parametrize("heads", [1, 3, 8])
@pytest.mark.parametrize("fmt", ["turbo2", "turbo3", "turbo4"])
def test_odd_rows_of_long_appends(fmt, heads, norm_correction, dtype):
    import torch
    import turboquant_plus_b200 as tq
    vectors = PAIR * torch.cuda.get_device_properties(0).multi_processor_count
    tokens = -(-vectors // heads) + 5
    gen = torch.Generator(device="cuda").manual_seed(heads)
    rows = [_odd_rows(tokens, heads, dtype, gen) for _ in range(2)]
    n_pages = -(-tokens // 128)
    slots = torch.arange(tokens, device="cuda")
    got = []
    for piece in (tokens, 1000):
        cache = tq.PagedKVCache(D, heads, n_pages, 128, fmt, fmt, seed=42, norm_correction=norm_correction)
        cache.pool.zero_()
        for lo in range(0, tokens, piece):
            cache.append(rows[0][lo:lo + piece], rows[1][lo:lo + piece], slots[lo:lo + piece])
        got.append(_fields(cache))
    a, b = got
    for t in ("k", "v"):
        assert torch.equal(a[t], b[t])
        sa, sb = a[t + "_scale"], b[t + "_scale"]
        assert bool((((sa - sb).abs() <= 6 * 2.0 ** -24 * sb.abs()) | (sa == sb) | (sa.isnan() & sb.isnan())).all())


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("norm_correction", [True, False])
@pytest.mark.parametrize("fmt,heads", [("prod3", 1), ("prod3", 8), ("prod4", 3)])
def test_odd_rows_of_long_appends_of_keys_with_a_sketch(fmt, heads, norm_correction, dtype):
    """Every bit of the records, zero residuals and projections, rows at the type's ends, beyond its range and not finite ones among them."""
    import torch
    import turboquant_plus_b200 as tq
    tokens = -(-SKETCH * torch.cuda.get_device_properties(0).multi_processor_count // heads) + 5
    gen = torch.Generator(device="cuda").manual_seed(heads)
    rows = _odd_rows(tokens, heads, dtype, gen)
    n_pages = -(-tokens // 128)
    slots = torch.arange(tokens, device="cuda")
    got = []
    for piece in (tokens, 1000):
        cache = tq.PagedKVCache(D, heads, n_pages, 128, fmt, "turbo2", seed=42, norm_correction=norm_correction)
        cache.pool.zero_()
        for lo in range(0, tokens, piece):
            cache.append(rows[lo:lo + piece], rows[lo:lo + piece], slots[lo:lo + piece])
        got.append(_fields(cache))
    a, b = got
    assert {"k", "k_scale", "k_sketch", "k_rscale"} <= set(a)
    for name in a:
        if name.startswith("k"):
            assert torch.equal(a[name].contiguous().view(torch.uint8), b[name].contiguous().view(torch.uint8)), name


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("bits,norm_correction,width", [(2, True, 128), (3, True, 136), (3, False, 128), (4, True, 256), (4, False, 136)])
def test_long_packed_arrays(bits, norm_correction, width, dtype):
    """Packed indices, norms and factors as plain arrays, rows with elements between them."""
    import torch
    import turboquant_plus_b200 as tq
    n = ALONE * torch.cuda.get_device_properties(0).multi_processor_count + 77
    gen = torch.Generator(device="cuda").manual_seed(n + bits)
    rows = torch.full((n, width), float("nan"), device="cuda", dtype=getattr(torch, dtype))
    rows[:, :D] = _odd_rows(n, 1, dtype, gen)[:, 0]
    q = tq.PolarQuant(D, bits, seed=3, norm_correction=norm_correction, rotation="wht")
    whole = q.quantize_device(rows, packed=True, want_scale=True)
    few = [q.quantize_device(rows[lo:lo + 50000], packed=True, want_scale=True) for lo in range(0, n, 50000)]
    assert torch.equal(whole["packed"], torch.cat([f["packed"] for f in few]))
    for name, roundings in (("norm", 0), ("scale", 6)):
        a, b = whole[name], torch.cat([f[name] for f in few])
        assert bool((((a - b).abs() <= roundings * 2.0 ** -24 * b.abs()) | (a == b) | (a.isnan() & b.isnan())).all())


def test_captured_by_a_new_thread():
    """A long append whose first call in a thread is captured there."""
    import threading

    import torch
    import turboquant_plus_b200 as tq
    heads = 8
    tokens = PAIR * torch.cuda.get_device_properties(0).multi_processor_count // heads + 1
    n_pages = -(-tokens // 128)
    gen = torch.Generator(device="cuda").manual_seed(1)
    k, v = (torch.randn(tokens, heads, D, device="cuda", generator=gen).half() for _ in range(2))
    slots = torch.arange(tokens, device="cuda")
    caches = [tq.PagedKVCache(D, heads, n_pages, 128, "turbo3", "turbo3", seed=42) for _ in range(2)]
    for cache in caches:
        cache.pool.zero_()
        cache.append(k[:1], v[:1], slots[:1])                       # (constants on the device)
    torch.cuda.synchronize()
    graph, failed = torch.cuda.CUDAGraph(), []

    def work():
        try:
            with torch.cuda.graph(graph):
                caches[0].append(k, v, slots)
        except Exception as e:                                      # noqa: BLE001
            failed.append(e)

    thread = threading.Thread(target=work)
    thread.start()
    thread.join()
    assert not failed, failed
    graph.replay()
    caches[1].append(k, v, slots)
    torch.cuda.synchronize()
    assert torch.equal(caches[0].pool, caches[1].pool)
    graph.reset()
