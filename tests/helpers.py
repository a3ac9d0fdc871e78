"""Helpers shared by the GPU parity tests."""
import numpy as np

from oracle import tq_oracle as o

D = 128


def boundary_band(c):
    """Half-width of the band around a decision boundary inside which an index may differ from the
    fp64 reference: 1e-6 relative to the largest centroid magnitude."""
    return 1e-6 * np.abs(c).max()


def near_boundary(y, c):
    """Boolean mask: rotated coordinate within the band of some boundary."""
    b = o.boundaries(c)
    return (np.abs(y[..., None] - b).min(axis=-1) <= boundary_band(c))


def check_indices(idx_gpu, idx_ref, y_ref, c):
    """Indices equal except inside the boundary band; returns (mismatches, coordinates in band)."""
    diff = idx_gpu != idx_ref
    band = near_boundary(y_ref, c)
    assert not (diff & ~band).any(), f"{int((diff & ~band).sum())} index mismatches outside the boundary band"
    assert (np.abs(idx_gpu.astype(np.int64) - idx_ref.astype(np.int64))[diff] <= 1).all()
    return int(diff.sum()), int(band.sum())


def max_rel(out, ref):
    """Max-relative error per row: max|out-ref| / max|ref|, worst row."""
    out = np.asarray(out, dtype=np.float64).reshape(-1, out.shape[-1])
    ref = np.asarray(ref, dtype=np.float64).reshape(-1, ref.shape[-1])
    return float((np.abs(out - ref).max(axis=1) / np.abs(ref).max(axis=1)).max())


def wht_dense(c, seed):
    return o.wht_as_dense(c[f"wht_s1_{seed}"], c[f"wht_s2_{seed}"])


def fill_cache(cache, k, v, seq_lens, rng, page_tokens=128):
    """Append per-sequence K/V (lists of (len, Hkv, d) arrays) into randomly chosen pages; returns
    the block table."""
    import torch
    n_pages = [(int(n) + page_tokens - 1) // page_tokens for n in seq_lens]
    perm = rng.permutation(cache.num_pages)[: sum(n_pages)]
    max_pages = max(n_pages)
    bt = np.zeros((len(seq_lens), max_pages), dtype=np.int32)
    pos = 0
    for b, n in enumerate(seq_lens):
        pages = perm[pos:pos + n_pages[b]]
        pos += n_pages[b]
        bt[b, : n_pages[b]] = pages
        t = np.arange(int(n))
        slots = pages[t // page_tokens].astype(np.int64) * page_tokens + t % page_tokens
        cache.append(torch.as_tensor(k[b]).to(cache.device), torch.as_tensor(v[b]).to(cache.device),
                     torch.as_tensor(slots))
    return torch.as_tensor(bt)


def stored_rows(cache, which, pages, n):
    """(n, heads, D) fp64 rows that a cache holds for a sequence, decoded from its records in plain NumPy: what attention has
    to see, whichever neighbouring index a coordinate on a decision boundary took when it was quantized."""
    lay, pt = cache.layout, cache.page_tokens
    fmt = cache.k_format if which == "k" else cache.v_format
    pool = cache.pool[np.asarray(pages, dtype=np.int64)].cpu().numpy()           # (pages, heads, record)

    def field(off, per_token, dtype):
        a = np.ascontiguousarray(pool[:, :, off:off + pt * per_token]).view(dtype)
        return a.reshape(pool.shape[0], pool.shape[1], pt, -1).transpose(0, 2, 1, 3).reshape(-1, pool.shape[1], a.shape[2] // pt)[:n]

    idx = field(getattr(lay, which + "_idx_off"), getattr(lay, which + "_idx_bytes"), np.uint8)
    if fmt == "q8_0":
        scale = field(getattr(lay, which + "_scale_off"), 8, np.float16).astype(np.float64)
        return idx.view(np.int8).astype(np.float64) * np.repeat(scale, 32, axis=2)
    quant = cache.k_quantizer if which == "k" else cache.v_quantizer
    prod = fmt.startswith("prod")
    pq = quant.polar_quant if prod else quant
    bits = np.unpackbits(idx, axis=2).reshape(*idx.shape[:2], D, pq.bit_width)
    codes = (bits * (1 << np.arange(pq.bit_width - 1, -1, -1))).sum(axis=3)
    scale = field(getattr(lay, which + "_scale_off"), 4, np.float32).astype(np.float64)
    rows = (pq.centroids[codes] @ pq.rotation) * scale
    if prod:
        signs = 2.0 * np.unpackbits(field(lay.k_qjl_off, D // 8, np.uint8), axis=2) - 1.0
        rows = rows + (signs @ quant.qjl.S) * field(lay.k_rscale_off, 4, np.float32).astype(np.float64)
    return rows
