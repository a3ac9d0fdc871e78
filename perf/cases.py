"""Cases that stand for what a program does with the compressed KV cache, each one pass through the public entry points:

  decode    a decode step of a model: per layer the new token of every sequence is appended (quantized), then attended
  step      the same for a whole stack of layers from pinned host buffers (``LayeredKVCache.decode_step``)
  prefill   a chunk of new positions is appended to one layer's cache, then attends causally to the prefix and itself
  append    a prompt's K and V rows are quantized into the pages of one layer
  vectors   the library calls of the reference's API: ``quantize`` then ``dequantize`` of a batch of vectors
  compress  ``KVCacheCompressor.compress`` then ``decompress`` of whole K and V tensors

Shapes are those of the benchmark configurations (32 / 8 and 64 / 8 heads of 128, KV-head shards of them, 128-token
pages, contexts up to 131,072).  Keys are N(0,1) with a lognormal scale per vector, four outlier channels and a
RoPE-style rotation by position; values and queries are N(0,1).
"""
from __future__ import annotations

import math

import torch

import turboquant_plus_b200 as tq
from turboquant_plus_b200.layered import LayeredKVCache, boundary_format_table

D, PAGE = 128, 128
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
CHUNK = 131072          # tokens whose K and V rows are made at a time while a cache is filled


def listed():
    return [
        # the first tokens of a chat: one short sequence, an eager loop over layers, the default call
        {"name": "decode-chat", "kind": "decode", "layers": 2, "batch": 1, "ctx": 517, "ragged": False, "hq": 32, "hkv": 8,
         "k": "turbo3", "v": "turbo3", "dtype": "f16", "overlap": False},
        # one sequence at 32K tokens through the whole stack, host buffers in and out
        {"name": "step-32k", "kind": "step", "layers": 40, "batch": 1, "ctx": 32768, "hq": 32, "hkv": 8,
         "k": "turbo3", "v": "turbo3", "keep": 0, "dtype": "f16"},
        # batched decode of a stack with 8-bit keys, 2-bit values and boundary layers at 8 bits
        {"name": "step-batch16-asym", "kind": "step", "layers": 32, "batch": 16, "ctx": 8192, "hq": 32, "hkv": 8,
         "k": "q8_0", "v": "turbo2", "keep": 2, "dtype": "f16"},
        # a serving batch of unequal sequences, keys with the sign sketch
        {"name": "decode-ragged256", "kind": "decode", "layers": 1, "batch": 256, "ctx": 32768, "ragged": True, "hq": 32,
         "hkv": 8, "k": "prod3", "v": "turbo3", "dtype": "f16", "overlap": "append"},
        # long-context decode with eight query heads per KV head
        {"name": "decode-gqa8-128k", "kind": "decode", "layers": 1, "batch": 2, "ctx": 131072, "ragged": False, "hq": 64,
         "hkv": 8, "k": "turbo4", "v": "turbo4", "dtype": "bf16", "overlap": "append"},
        # the last chunk of a 128K prompt
        {"name": "prefill-128k", "kind": "prefill", "batch": 1, "chunk": 128, "ctx": 131072, "hq": 64, "hkv": 8,
         "k": "turbo3", "v": "turbo3", "dtype": "f16"},
        # a whole prompt of an odd length in one call
        {"name": "prefill-prompt", "kind": "prefill", "batch": 1, "chunk": 3999, "ctx": 3999, "hq": 32, "hkv": 8,
         "k": "turbo4", "v": "turbo3", "dtype": "bf16"},
        # chunks of two sequences over a cache with 8-bit keys and 2-bit values
        {"name": "prefill-asym", "kind": "prefill", "batch": 2, "chunk": 128, "ctx": 8192, "hq": 32, "hkv": 8,
         "k": "q8_0", "v": "turbo2", "dtype": "f16"},
        # a chunk of a prompt on its way into the cache
        {"name": "append-8k", "kind": "append", "tokens": 8192, "hkv": 8, "k": "turbo3", "v": "turbo3", "dtype": "f16"},
        # a long prompt, keys with the sign sketch
        {"name": "append-128k-prod", "kind": "append", "tokens": 131072, "hkv": 8, "k": "prod3", "v": "turbo3",
         "dtype": "bf16"},
        # the reference's round trip: NumPy in, NumPy out, the default rotation
        {"name": "vectors-numpy", "kind": "vectors", "n": 65536, "quantizer": "mse", "bits": 3, "rotation": "dense",
         "host": True, "dtype": "f32"},
        # K and V of a few layers through the compressor on the device, the default rotation
        {"name": "compress-cuda", "kind": "compress", "layers": 4, "hkv": 8, "seq": 2000, "k_bits": 3, "v_bits": 3,
         "rotation": "dense", "host": False, "dtype": "f16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


FORMATS = [("turbo3", "turbo3"), ("turbo3", "turbo3"), ("turbo4", "turbo4"), ("turbo2", "turbo2"), ("turbo4", "turbo3"),
           ("q8_0", "turbo2"), ("prod3", "turbo3"), ("prod4", "turbo4")]
HEADS = [(32, 8), (32, 8), (64, 8), (16, 4), (16, 2), (4, 1)]     # whole models and KV-head shards of them


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "step", "prefill", "prefill", "append", "append", "vectors",
                       "vectors", "compress"])
    k, v = rng.choice(FORMATS)
    hq, hkv = rng.choice(HEADS)
    dtype = rng.choice(["f16", "f16", "bf16"])
    if kind == "decode":
        batch = _log_int(rng, 1, 256)
        layers = rng.choice([1, 1, 2, 4])
        most = min(131072, 4_000_000 // (batch * layers))         # cached positions of the largest listed case
        return {"kind": kind, "layers": layers, "batch": batch, "ctx": _log_int(rng, 64, most),
                "ragged": batch > 1 and rng.random() < 0.6, "hq": hq, "hkv": hkv, "k": k, "v": v, "dtype": dtype,
                "overlap": rng.choice([False, "append"])}
    if kind == "step":
        batch, layers = _log_int(rng, 1, 32), rng.randint(4, 40)
        most = min(32768, 3_000_000 // (batch * layers))
        return {"kind": kind, "layers": layers, "batch": batch, "ctx": _log_int(rng, 128, most), "hq": hq, "hkv": hkv,
                "k": k, "v": v, "keep": rng.choice([0, 2]) if k == "q8_0" else 0, "dtype": dtype}
    if kind == "prefill":
        chunk, batch = _log_int(rng, 16, 4096), rng.choice([1, 1, 2, 4])
        most = max(chunk, min(131072, 128 * 131072 // (chunk * batch)))
        return {"kind": kind, "batch": batch, "chunk": chunk, "ctx": max(chunk, _log_int(rng, 128, max(most, 129))),
                "hq": hq, "hkv": hkv, "k": k, "v": v, "dtype": dtype}
    if kind == "append":
        return {"kind": kind, "tokens": _log_int(rng, 1, 131072), "hkv": hkv, "k": k, "v": v,
                "dtype": rng.choice(["f16", "f16", "bf16", "f32"])}
    rotation = rng.choice(["dense", "wht"])
    host = rng.random() < 0.5
    dtype = "f32" if host else rng.choice(["f32", "f16"])
    if kind == "vectors":
        quantizer = rng.choice(["mse", "prod"])
        return {"kind": kind, "n": _log_int(rng, 1, 65536), "quantizer": quantizer,
                "bits": rng.randint(2, 4), "rotation": rotation, "host": host, "dtype": dtype}
    return {"kind": kind, "layers": rng.randint(1, 8), "hkv": rng.choice([1, 2, 4, 8]), "seq": _log_int(rng, 16, 1000),
            "k_bits": rng.randint(2, 4), "v_bits": rng.randint(2, 4), "rotation": rotation, "host": host, "dtype": dtype}


# ---- inputs -----------------------------------------------------------------------------------------
class _Source:
    """Keys, values and queries of one seed, made on the device."""

    def __init__(self, seed):
        self.dev = torch.device("cuda", torch.cuda.current_device())
        self.gen = torch.Generator(device=self.dev)
        self.gen.manual_seed(seed)
        self.outliers = torch.randperm(D, generator=self.gen, device=self.dev)[:4]
        self.freq = 10000.0 ** (-torch.arange(0, D, 2, device=self.dev, dtype=torch.float32) / D)

    def normal(self, *shape, dtype=torch.float32):
        return torch.randn(shape, generator=self.gen, device=self.dev, dtype=torch.float32).to(dtype)

    def perm(self, n):
        return torch.randperm(n, generator=self.gen, device=self.dev)

    def keys(self, positions, heads, dtype):
        """(len(positions), heads, D)"""
        k = self.normal(positions.numel(), heads, D)
        k *= torch.exp(0.5 * self.normal(positions.numel(), heads, 1))
        k[:, :, self.outliers] *= 10.0
        ang = positions.to(torch.float32)[:, None, None] * self.freq
        rot = torch.polar(torch.ones_like(ang), ang)
        return torch.view_as_real(torch.view_as_complex(k.view(*k.shape[:2], D // 2, 2)) * rot).reshape(k.shape).to(dtype)

    def values(self, n, heads, dtype):
        return self.normal(n, heads, D, dtype=dtype)


def _lengths(case, src):
    """Cached positions per sequence, the last token (or chunk) included."""
    batch, ctx = case["batch"], case["ctx"]
    if not case.get("ragged"):
        return [ctx] * batch
    lo = max(1, ctx // 32)                   # evenly spread over [ctx / 32, ctx], in an order of the seed's own
    return [lo + (ctx - lo) * i // (batch - 1) for i in src.perm(batch).tolist()]


def _pages(lengths, src):
    """A shuffled block table (batch, most pages) and the number of pages in use."""
    n_pages = [-(-n // PAGE) for n in lengths]
    table = torch.zeros((len(lengths), max(n_pages)), dtype=torch.int32)
    perm, at = src.perm(sum(n_pages)).to(torch.int32).cpu(), 0
    for b, n in enumerate(n_pages):
        table[b, :n] = perm[at:at + n]
        at += n
    return table.to(src.dev), sum(n_pages)


def _positions(lengths, table, dev):
    """Position and slot of every cached token, sequence after sequence."""
    n = torch.tensor(lengths, device=dev)
    seq = torch.repeat_interleave(torch.arange(len(lengths), device=dev), n)
    pos = torch.arange(int(n.sum()), device=dev) - torch.repeat_interleave(torch.cumsum(n, 0) - n, n)
    return pos, table[seq, pos // PAGE].to(torch.int64) * PAGE + pos % PAGE


def _slots_from(starts, count, table, dev):
    """Slots of ``count`` tokens of every sequence from ``starts`` on, (batch * count,)."""
    pos = torch.tensor(starts, device=dev)[:, None] + torch.arange(count, device=dev)[None, :]
    return (torch.gather(table.to(torch.int64), 1, pos // PAGE) * PAGE + pos % PAGE).reshape(-1)


def _fill(append, lengths, table, heads, dtype, src):
    pos, slots = _positions(lengths, table, src.dev)
    for lo in range(0, pos.numel(), CHUNK):
        p = pos[lo:lo + CHUNK]
        append(src.keys(p, heads, dtype), src.values(p.numel(), heads, dtype), slots[lo:lo + CHUNK])


def _records(cache):
    """The arrays that make up a cache's pages, as views of its pool."""
    lay, pool = cache.layout, cache.pool

    def array(off, per_token, dtype=torch.uint8):
        return pool[..., off:off + PAGE * per_token].view(dtype)

    out = {}
    for t, fmt in (("k", cache.k_format), ("v", cache.v_format)):
        out[t] = array(getattr(lay, t + "_idx_off"), getattr(lay, t + "_idx_bytes"))
        q8 = fmt == "q8_0"
        out[t + "_scale"] = array(getattr(lay, t + "_scale_off"), 8 if q8 else 4, torch.float16 if q8 else torch.float32)
        if fmt.startswith("prod"):
            out[t + "_sketch"] = array(lay.k_qjl_off, D // 8)
            out[t + "_rscale"] = array(lay.k_rscale_off, 4, torch.float32)
    return out


def _formats(case):
    pair = (case["k"], case["v"])
    if case.get("keep"):
        return boundary_format_table(case["layers"], pair, ("q8_0", "q8_0"), keep=case["keep"])
    return [pair] * case["layers"]


def _prepare_decode(case, src):
    dt, L, B, hq, hkv = DTYPES[case["dtype"]], case["layers"], case["batch"], case["hq"], case["hkv"]
    lengths = _lengths(case, src)
    table, n_pages = _pages(lengths, src)
    cache = LayeredKVCache(L, D, hkv, n_pages, PAGE, _formats(case), seed=42)
    for layer in range(L):
        _fill(lambda k, v, s: cache.append(layer, k, v, s), lengths, table, hkv, dt, src)
    last = torch.tensor(lengths, device=src.dev) - 1
    st = {"case": case, "cache": cache, "table": table, "lens": torch.tensor(lengths, dtype=torch.int32, device=src.dev),
          "slots": _slots_from(last.tolist(), 1, table, src.dev),
          "q": [src.normal(B, hq, D, dtype=dt) for _ in range(L)],
          "k": [src.keys(last, hkv, dt) for _ in range(L)], "v": [src.values(B, hkv, dt) for _ in range(L)],
          "out": [torch.empty((B, hq, D), dtype=dt, device=src.dev) for _ in range(L)],
          "workspace": cache.layers[0].workspace(B, hq, table.shape[1])}
    st["records"] = [_records(whole) for whole, _ in cache.groups]
    return st


def _run_decode(st):
    cache, table, lens, slots, overlap = st["cache"], st["table"], st["lens"], st["slots"], st["case"]["overlap"]
    for i in range(cache.num_layers):
        cache.append(i, st["k"][i], st["v"][i], slots)
        cache.attend(i, st["q"][i], table, lens, out=st["out"][i], workspace=st["workspace"], overlap=overlap)
    return {"out": st["out"], "records": st["records"]}


def _prepare_step(case, src):
    dt, L, B, hq, hkv = DTYPES[case["dtype"]], case["layers"], case["batch"], case["hq"], case["hkv"]
    lengths = [case["ctx"]] * B
    table, n_pages = _pages([n + 1 for n in lengths], src)              # a place for the step's token
    cache = LayeredKVCache(L, D, hkv, n_pages, PAGE, _formats(case), seed=42)
    for layer in range(L):
        _fill(lambda k, v, s: cache.append(layer, k, v, s), lengths, table, hkv, dt, src)
    lens = torch.tensor(lengths, dtype=torch.int32, device=src.dev)
    step = cache.prepare_decode(B, hq, table, lens, dtype=dt)
    q, k, v, out = cache.host_buffers()
    pos = torch.full((L * B,), case["ctx"], device=src.dev)
    q.copy_(src.normal(L, B, hq, D, dtype=dt))
    k.copy_(src.keys(pos, hkv, dt).view(L, B, hkv, D))
    v.copy_(src.values(L * B, hkv, dt).view(L, B, hkv, D))
    return {"case": case, "cache": cache, "step": step, "lens": lens, "host": (q, k, v, out),
            "records": [_records(whole) for whole, _ in cache.groups]}


def _run_step(st):
    st["step"]["len"].copy_(st["lens"])          # the lengths of this step, as the scheduler has them
    out = st["cache"].decode_step(*st["host"])
    return {"out": out, "records": st["records"]}


def _prepare_prefill(case, src):
    dt, B, chunk, hq, hkv = DTYPES[case["dtype"]], case["batch"], case["chunk"], case["hq"], case["hkv"]
    lengths = [case["ctx"]] * B
    table, n_pages = _pages(lengths, src)
    cache = tq.PagedKVCache(D, hkv, n_pages, PAGE, case["k"], case["v"], seed=42)
    _fill(cache.append, lengths, table, hkv, dt, src)
    first = case["ctx"] - chunk
    pos = (first + torch.arange(chunk, device=src.dev)).repeat(B)
    return {"case": case, "cache": cache, "table": table, "lens": torch.tensor(lengths, dtype=torch.int32, device=src.dev),
            "k": src.keys(pos, hkv, dt), "v": src.values(B * chunk, hkv, dt), "q": src.normal(B, chunk, hq, D, dtype=dt),
            "slots": _slots_from([first] * B, chunk, table, src.dev), "records": _records(cache)}


def _run_prefill(st):
    st["cache"].append(st["k"], st["v"], st["slots"])
    out = st["cache"].prefill_attend(st["q"], st["table"], st["lens"])
    return {"out": out, "records": st["records"]}


def _prepare_append(case, src):
    dt, n, hkv = DTYPES[case["dtype"]], case["tokens"], case["hkv"]
    table, n_pages = _pages([n], src)
    cache = tq.PagedKVCache(D, hkv, n_pages, PAGE, case["k"], case["v"], seed=42)
    pos, slots = _positions([n], table, src.dev)
    return {"case": case, "cache": cache, "slots": slots, "k": src.keys(pos, hkv, dt), "v": src.values(n, hkv, dt),
            "records": _records(cache)}


def _run_append(st):
    st["cache"].append(st["k"], st["v"], st["slots"])
    return st["records"]


def _prepare_vectors(case, src):
    kind = tq.TurboQuantMSE if case["quantizer"] == "mse" else tq.TurboQuant
    quantizer = kind(D, case["bits"], seed=42, rotation=case["rotation"])
    x = src.keys(torch.arange(case["n"], device=src.dev), 1, DTYPES[case["dtype"]]).reshape(case["n"], D)
    return {"case": case, "quantizer": quantizer, "x": x.cpu().numpy() if case["host"] else x}


def _run_vectors(st):
    quantizer = st["quantizer"]
    if st["case"]["quantizer"] == "mse":
        indices, norms = quantizer.quantize(st["x"])
        return {"indices": indices, "norms": norms, "x_hat": quantizer.dequantize(indices, norms)}
    code = quantizer.quantize(st["x"])
    return {"indices": code.mse_indices, "norms": code.vector_norms, "signs": code.qjl_signs,
            "residual_norms": code.residual_norms, "x_hat": quantizer.dequantize(code)}


def _prepare_compress(case, src):
    dt, shape = DTYPES[case["dtype"]], (case["layers"], case["hkv"], case["seq"], D)
    comp = tq.KVCacheCompressor(D, k_bits=case["k_bits"], v_bits=case["v_bits"], seed=42, rotation=case["rotation"])
    pos = torch.arange(case["seq"], device=src.dev).repeat(case["layers"] * case["hkv"])
    k, v = src.keys(pos, 1, dt).reshape(shape), src.values(pos.numel(), 1, dt).reshape(shape)
    if case["host"]:
        k, v = k.cpu().numpy(), v.cpu().numpy()
    return {"case": case, "compressor": comp, "k": k, "v": v}


def _run_compress(st):
    comp = st["compressor"]
    return comp.decompress(comp.compress(st["k"], st["v"]))        # (K, V): every code and norm goes into them


_PREPARE = {"decode": _prepare_decode, "step": _prepare_step, "prefill": _prepare_prefill, "append": _prepare_append,
            "vectors": _prepare_vectors, "compress": _prepare_compress}
_RUN = {"decode": _run_decode, "step": _run_step, "prefill": _run_prefill, "append": _run_append,
        "vectors": _run_vectors, "compress": _run_compress}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, _Source(seed))


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ---- what a pass cannot do without -------------------------------------------------------------------
def _vector_bytes(fmt):
    """Bytes of one stored vector."""
    if fmt == "q8_0":
        return D + D // 32 * 2
    bits = int(fmt[-1])
    return 16 * bits + 4 + (4 if fmt.startswith("prod") else 0)


def _row_bytes(case):
    return D * (4 if case["dtype"] == "f32" else 2)


def work(case):
    kind = case["kind"]
    if kind in ("decode", "step"):
        B, L, hkv, hq = case["batch"], case["layers"], case["hkv"], case["hq"]
        tokens = B * case["ctx"] * (0.5 + 1 / 64 if case.get("ragged") else 1.0)
        cached = sum(_vector_bytes(k) + _vector_bytes(v) for k, v in _formats(case))
        new = L * B * (2 * hkv + 2 * hq) * _row_bytes(case) + B * hkv * cached
        return {"bytes": tokens * hkv * cached + new, "flops": 4.0 * L * tokens * hq * D}
    if kind == "prefill":
        B, n, ctx, hkv, hq = case["batch"], case["chunk"], case["ctx"], case["hkv"], case["hq"]
        pair = _vector_bytes(case["k"]) + _vector_bytes(case["v"])
        seen = n * (ctx - n) + n * (n + 1) / 2                          # (query, visible position) pairs
        return {"bytes": B * (ctx * hkv * pair + n * ((2 * hkv + 2 * hq) * _row_bytes(case))), "flops": 4.0 * B * hq * D * seen}
    if kind == "append":
        vectors = case["tokens"] * case["hkv"]
        return {"bytes": vectors * (2 * _row_bytes(case) + _vector_bytes(case["k"]) + _vector_bytes(case["v"])),
                "flops": 2.0 * vectors * D * 7}
    n = case["n"] if kind == "vectors" else case["layers"] * case["hkv"] * case["seq"]
    turn = 2.0 * D * D if case["rotation"] == "dense" else 7.0 * D      # one rotation of one vector
    index = 8 if case["host"] else 1
    back = 8 if case["host"] or case["rotation"] == "dense" else 4
    mse = {"bytes": n * (_row_bytes(case) + D * (2 * index + back)), "flops": n * 2 * turn}
    prod = {"bytes": n * (_row_bytes(case) + D * (2 * index + 2 + back)), "flops": n * 5 * turn}
    if kind == "vectors":
        return mse if case["quantizer"] == "mse" else prod
    return {m: mse[m] + prod[m] for m in mse}


def tolerance(case):
    kind = case["kind"]
    if kind in ("vectors", "compress"):
        if case["rotation"] == "dense":
            return {"rel": 1e-6, "differ": 1e-6}                        # 64-bit sums, norms in 32 bits
        # 32-bit sums: a coordinate on a decision boundary may take the neighbouring level, one in some millions
        return {"rel": 1e-3, "max": 0.99, "differ": 1e-5}
    if kind == "append":
        return {"rel": 1e-5, "max": 0.1, "differ": 1e-5}                # scales in 32 bits, indices as above
    # 16-bit operands with 32-bit sums, results in the queries' type
    return {"rel": 8e-3 if case["dtype"] == "bf16" else 2e-3, "differ": 1e-5}
