"""Dense-mode calls of many vectors (integer products of base-256 digits) against the same vectors in small calls (fp64 products):
edges of the 128-vector tiles, both row types, all widths, rows that are zero, tiny, huge or not finite, matrices that are not
rotations (uneven ones stay with the fp64 products).  Both paths are within 7e-16 of exact sums, so indices and signs are equal except within 1e-14 of a boundary, which
these inputs do not meet; reconstructions agree to 256 roundings of 2^-53 of the largest one of their row (sums of 256 terms)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
D = 128
PIECE = 4096          # small calls


def _pieces(fn, x):
    import torch
    parts = [fn(x[lo:lo + PIECE]) for lo in range(0, len(x), PIECE)]
    return [torch.cat(p) for p in zip(*parts)]


def _same(a, b):
    import torch
    return bool(((a == b) | (torch.isnan(a) & torch.isnan(b))).all()) if a.is_floating_point() else torch.equal(a, b)


def _rows(n, dtype, special):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, D, device="cuda", generator=gen) * torch.exp(0.5 * torch.randn(n, 1, device="cuda", generator=gen))
    x[:, 5] *= 10
    x[n // 2] = 0
    if special:
        big, small = (1e30, 1e-30) if dtype == "float32" else (6e4, 1e-7)
        x[3] = 0
        x[3, 7] = small
        x[4] = big
        x[9] *= small
        x[10, 3], x[11, 3], x[n - 1, 0] = float("nan"), float("inf"), float("-inf")
        x[129, 100], x[130, 100] = float("inf"), float("-inf")
    return x.to(getattr(torch, dtype))


@pytest.mark.parametrize("dtype", ["float32", "float16"])
@pytest.mark.parametrize("n,bits,special", [(9473, 2, False), (9600, 3, True), (9601, 4, False), (18944, 3, False), (19073, 2, True), (40000, 4, True)])
@pytest.mark.parametrize("matrix", ["rotation", "arbitrary", "long"])
def test_many_vectors_equal_few(n, bits, special, dtype, matrix):
    import torch
    import turboquant_plus_b200 as tq
    x = _rows(n, dtype, special)
    q = tq.TurboQuant(D, bits, seed=5)          # bits - 1 for the indices, one for the sketch
    m = tq.TurboQuantMSE(D, bits, seed=6)
    if matrix == "arbitrary":                   # residuals of many times the vector's length
        rng = np.random.default_rng(n)
        q.polar_quant.rotation = rng.standard_normal((D, D)) * np.exp(rng.standard_normal((D, D)))
        m.polar_quant.rotation = np.diag(np.exp2(rng.integers(-20, 20, D).astype(float)))
    if matrix == "long":                        # the same from matrices whose entries are of one size, which have digits
        rng = np.random.default_rng(n)
        q.polar_quant.rotation, m.polar_quant.rotation = 3 * rng.standard_normal((D, D)), rng.standard_normal((D, D))

    def quantize(v):
        c = q.quantize(v)
        return c.mse_indices, c.vector_norms, c.qjl_signs, c.residual_norms

    whole, parts = quantize(x), _pieces(quantize, x)
    assert _same(whole[0], parts[0]) and _same(whole[1], parts[1])
    finite = torch.isfinite(parts[3])
    assert torch.equal(torch.isfinite(whole[3]), finite)
    assert bool(((whole[3] - parts[3]).abs() <= 1.2e-7 * parts[3])[finite].all())          # fp32 results of sums that agree
    if matrix == "rotation":                    # (otherwise: projections of any size beside others, signs within rounding of zero)
        assert torch.equal(whole[2], parts[2])
    else:
        assert float((whole[2] != parts[2]).float().mean()) < 1e-6
    idx, norms = m.quantize(x)
    few = _pieces(m.quantize, x)
    assert _same(idx, few[0]) and _same(norms, few[1])

    def close(a, b):
        scale = b.abs().amax(dim=1, keepdim=True).nan_to_num(posinf=1.0)
        ok = ((a - b).abs() <= 256 * 2.0 ** -53 * scale) | (a == b) | (~torch.isfinite(a) & ~torch.isfinite(b))
        return bool(ok.all())

    code = q.quantize(x)
    back = q.dequantize(code)
    parts = torch.cat([q.dequantize(type(code)(**{f: (getattr(code, f)[lo:lo + PIECE] if torch.is_tensor(getattr(code, f)) else getattr(code, f))
                                                  for f in code.__dataclass_fields__})) for lo in range(0, n, PIECE)])
    assert close(back, parts)
    assert close(m.dequantize(idx, norms), torch.cat([m.dequantize(idx[lo:lo + PIECE], norms[lo:lo + PIECE]) for lo in range(0, n, PIECE)]))


def _uneven(kind, rng):
    """(rotation or None, S or None, centroids or None) that fixed-point digits of one scale do not carry to 53 bits."""
    r = np.linalg.qr(rng.standard_normal((D, D)))[0]
    s = rng.standard_normal((D, D))
    sizes = np.exp(rng.uniform(-40, 0, D))
    if kind == "rotation rows":
        return r * sizes[:, None], None, None
    if kind == "rotation columns":
        return r * sizes, None, None
    if kind == "sketch rows":
        return None, s * sizes[:, None], None
    if kind == "blocks":                        # outputs that see some of the elements only
        b = np.zeros((D, D))
        for lo in range(0, D, 16):
            b[lo:lo + 16, lo:lo + 16] = np.linalg.qr(rng.standard_normal((16, 16)))[0]
        return b, None, None
    return None, None, np.array([-1.0, -3e-9, 1e-9, 1.0])       # centroids


@pytest.mark.parametrize("kind", ["rotation rows", "rotation columns", "sketch rows", "blocks", "centroids"])
def test_uneven_constants(kind):
    """Matrices and codebooks whose entries differ much in size: many vectors as few, error held for every column, or row, by
    its own size (sums of 256 terms, as above)."""
    import torch
    import turboquant_plus_b200 as tq
    n = 9601
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, D, device="cuda", generator=gen)
    if kind == "blocks":
        x[:, 16:] *= 1e-20
    q = tq.TurboQuant(D, 3, seed=5)
    rot, s, cent = _uneven(kind, np.random.default_rng(n))
    if rot is not None:
        q.polar_quant.rotation = rot
    if s is not None:
        q.qjl.S = s
    if cent is not None:
        q.polar_quant.centroids = cent

    def quantize(v):
        c = q.quantize(v)
        return c.mse_indices, c.vector_norms, c.qjl_signs, c.residual_norms

    whole, parts = quantize(x), _pieces(quantize, x)
    assert torch.equal(whole[0], parts[0]) and torch.equal(whole[1], parts[1]) and torch.equal(whole[2], parts[2])
    pq = q.polar_quant
    idx, norms = whole[0], whole[1]
    if kind == "centroids":
        idx = 1 + (idx & 1)                     # the small ones only
    back = pq.dequantize(idx, norms)
    few = torch.cat([pq.dequantize(idx[lo:lo + PIECE], norms[lo:lo + PIECE]) for lo in range(0, n, PIECE)])
    size = few.abs().amax(dim=1 if kind == "centroids" else 0, keepdim=True)
    assert bool(((back - few).abs() <= 256 * 2.0 ** -53 * size).all())


def test_first_large_calls():
    """The first call of many vectors makes the digits: from several threads' streams at once, in a graph being captured (which
    takes the fp64 products), and in the direction of ``dequantize``."""
    import threading

    import torch
    import turboquant_plus_b200 as tq
    n, threads = 20011, 6
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, D, device="cuda", generator=gen)

    def fresh():
        q = tq.TurboQuant(D, 4, seed=9)
        q.quantize_device(x[:100])              # the constants are on the device, the digits are not
        return q

    def same(a, b):
        return all(torch.equal(a[name], b[name]) for name in b)

    right = fresh().quantize_device(x)
    for _ in range(3):
        q, got, start = fresh(), [None] * threads, threading.Barrier(threads)
        torch.cuda.synchronize()

        def work(i):
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                got[i] = q.quantize_device(x)
                torch.cuda.current_stream().synchronize()

        pool = [threading.Thread(target=work, args=(i,)) for i in range(threads)]
        [t.start() for t in pool]
        [t.join() for t in pool]
        assert all(same(g, right) for g in got)

    q, graph, other = fresh(), torch.cuda.CUDAGraph(), fresh()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        captured = q.quantize_device(x)
    graph.replay()
    torch.cuda.synchronize()
    assert same(captured, right) and same(q.quantize_device(x), right)
    graph.reset()

    code = other.quantize(x)
    back = fresh().dequantize(code)
    few = torch.cat([other.dequantize(type(code)(**{f: (getattr(code, f)[lo:lo + PIECE] if torch.is_tensor(getattr(code, f)) else getattr(code, f))
                                                     for f in code.__dataclass_fields__})) for lo in range(0, n, PIECE)])
    assert bool(((back - few).abs() <= 256 * 2.0 ** -53 * few.abs().amax(dim=1, keepdim=True)).all())


def _next_to_boundaries(quantizer, n, seed):
    """fp32 rows, some of whose rotated coordinates lie a relative 1e-9 to 1e-5 beside a decision boundary: one, a few or most of a row."""
    import torch
    rng = np.random.default_rng(seed)
    rot, cent = quantizer.rotation, quantizer.centroids
    bnd = (cent[1:] + cent[:-1]) / 2
    bnd = bnd[np.abs(bnd) > 1e-6]               # (beside the centre, what fp32 rows can hold)
    y = rng.standard_normal((n, D)) / np.sqrt(D)
    if len(bnd):
        near = rng.random((n, D)) < np.array([1 / D, 5 / D, 0.5])[np.arange(n) // 128 % 3][:, None]
        at = rng.choice(bnd, (n, D)) * (1 + rng.choice([-1, 1], (n, D)) * 10.0 ** rng.uniform(-9, -5, (n, D)))
        rest = 1 - (at ** 2 * near).sum(1)
        near[rest < 0.1] = False
        rest = np.where(rest < 0.1, 1, rest)
        y *= ~near
        y *= np.sqrt(rest / (y ** 2).sum(1))[:, None]
        y += at * near
    else:
        y[:, ::7] *= 1e-8
    x = (y @ rot) * np.exp(rng.standard_normal((n, 1)))
    x[5] = 0
    return torch.from_numpy(x.astype(np.float32)).cuda()


@pytest.mark.parametrize("bits", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [4737, 9601, 40000])
def test_outputs_next_to_boundaries(n, bits):
    """What the leading products cannot decide: by the deciding warp, by whole rows while its ring is full, and with the sketch."""
    import torch
    import turboquant_plus_b200 as tq
    m, q = tq.TurboQuantMSE(D, bits, seed=6), tq.TurboQuant(D, bits + 1, seed=6)
    x = _next_to_boundaries(m.polar_quant, n, 10 * n + bits)
    idx, norms = m.quantize(x)
    few = _pieces(m.quantize, x)
    assert torch.equal(idx, few[0]) and torch.equal(norms, few[1])
    scaled = m.polar_quant.quantize_device(x, want_scale=True)
    parts = torch.cat([m.polar_quant.quantize_device(x[lo:lo + PIECE], want_scale=True)["scale"] for lo in range(0, n, PIECE)])
    assert torch.equal(scaled["idx"], few[0]) and bool(((scaled["scale"] - parts).abs() <= 1.2e-7 * parts).all())

    def quantize(v):
        c = q.quantize(v)
        return c.mse_indices, c.vector_norms, c.qjl_signs, c.residual_norms

    whole, parts = quantize(x), _pieces(quantize, x)
    assert torch.equal(whole[0], parts[0]) and torch.equal(whole[1], parts[1]) and torch.equal(whole[2], parts[2])
    assert bool(((whole[3] - parts[3]).abs() <= 1.2e-7 * parts[3]).all())


def _nearest(quantizer, n, seed):
    """The random fp32 row of `n` with the output that is nearest to a boundary."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(n, D, device="cuda", generator=gen)
    bnd = torch.from_numpy((quantizer.centroids[1:] + quantizer.centroids[:-1]) / 2).cuda()
    y = (x / x.norm(dim=1, keepdim=True)).double() @ torch.from_numpy(quantizer.rotation).cuda().T
    return x[int((y[:, :, None] - bnd).abs().amin((1, 2)).argmin())]


@pytest.mark.parametrize("dtype", ["float32", "float16"])
@pytest.mark.parametrize("n,share", [(4737, 1.0), (20011, 1.0), (20011, 0.1), (40000, 0.02)])
def test_copies_of_a_close_vector(n, share, dtype):
    """Rows that all ask for fp64: every one of a tile, a part of the sixteen that are computed at a time, and one now and then."""
    import torch
    import turboquant_plus_b200 as tq
    m, q = tq.TurboQuantMSE(D, 3, seed=6), tq.TurboQuant(D, 4, seed=6)
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, D, device="cuda", generator=gen)
    x[torch.rand(n, device="cuda", generator=gen) < share] = _nearest(m.polar_quant, 200000, n)
    x = x.to(getattr(torch, dtype))
    if dtype == "float16":                          # (rounded, the row is no longer close; rows out of the norm's range ask for fp64 too)
        x[torch.rand(n, device="cuda", generator=gen) < share, 77] = float("inf")
    for of in (m, q):
        def quantize(v):
            out = of.quantize_device(v) if of is q else of.polar_quant.quantize_device(v, want_scale=True)
            return [out[name] for name in sorted(out)]
        whole, parts = quantize(x), _pieces(quantize, x)
        for a, b in zip(whole, parts):
            if a.is_floating_point():
                assert bool((((a - b).abs() <= 1.2e-7 * b.abs()) | (a == b) | (a.isnan() & b.isnan())).all())
            else:
                assert torch.equal(a, b)
    assert torch.equal(m.quantize(x)[0], torch.cat([m.quantize(x[lo:lo + PIECE])[0] for lo in range(0, n, PIECE)]))


@pytest.mark.parametrize("dtype", ["float32", "float16"])
@pytest.mark.parametrize("scale", [1e-7, 1e-5, 1e-3, 1e-2])
def test_small_residuals(scale, dtype):
    """Reconstructions quantized again, with noise of `scale` of their length: residuals from the rows' own rounding on.  Against small calls,
    whose fp64 sums are off by 4.9e-16 of the vector's length: of a residual, of which fp32 rows leave 2.6e-8 or more, 2e-8, and by an
    fp32 rounding of 6e-8 on both sides."""
    import torch
    import turboquant_plus_b200 as tq
    n = 20011
    gen = torch.Generator(device="cuda").manual_seed(n)
    q = tq.TurboQuant(D, 3, seed=6)
    x = torch.randn(n, D, device="cuda", generator=gen) * torch.exp(torch.randn(n, 1, device="cuda", generator=gen))
    code = q.polar_quant.quantize_device(x)
    y = q.polar_quant.dequantize_device(code["norm"], idx=code["idx"])
    y = (y + scale * y.norm(dim=1, keepdim=True) * torch.randn(n, D, device="cuda", generator=gen) / D ** 0.5).to(getattr(torch, dtype))

    def quantize(v):
        out = q.quantize_device(v)
        return out["idx"], out["norm"], out["qjl"], out["rnorm"]

    whole, parts = quantize(y), _pieces(quantize, y)
    assert torch.equal(whole[0], parts[0]) and torch.equal(whole[1], parts[1]) and torch.equal(whole[2], parts[2])
    assert float(((whole[3] - parts[3]).abs() / parts[3]).max()) <= 1.6e-7


@pytest.mark.parametrize("width,column", [(256, 0), (256, 128), (130, 2), (257, 1), (129, 0)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_results_into_columns_of_wider_rows(width, column, accumulate):
    """fp64 results beside, or added to, what wider rows hold: by tiled copies where base and rows are on 16 bytes, else by stores; a last tile
    whose rows end within a warp's 32."""
    import torch
    import turboquant_plus_b200 as tq
    from turboquant_plus_b200 import _native as nv
    n = 9473 + 128 * 148 + 39
    gen = torch.Generator(device="cuda").manual_seed(n + width)
    q = tq.TurboQuantMSE(D, 3, seed=6).polar_quant
    code = q.quantize_device(torch.randn(n, D, device="cuda", generator=gen))
    held = torch.randn(n + 1, width, device="cuda", generator=gen, dtype=torch.float64)
    handle, got = q._native(held.device).handle, []
    for piece in (n, PIECE):
        out = held.clone()
        for lo in range(0, n, piece):
            m = min(piece, n - lo)
            nv.call("tq_dequantize_strided", handle, nv.ptr(code["idx"][lo:lo + m]), nv.ptr(code["norm"][lo:lo + m]), m, nv.ptr(out[lo:, column:]),
                    width, accumulate, nv.stream_ptr())
        got.append(out)
    whole, few = got
    rest = torch.ones(n + 1, width, dtype=torch.bool, device="cuda")
    rest[:n, column:column + D] = False
    assert torch.equal(whole[rest], held[rest])
    a, b = whole[:n, column:column + D], few[:n, column:column + D]
    assert not torch.equal(a, held[:n, column:column + D])
    assert bool(((a - b).abs() <= 256 * 2.0 ** -53 * b.abs().amax(dim=1, keepdim=True)).all())
