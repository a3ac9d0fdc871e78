"""Chunked prefill by pairs of CTAs: one, two, three and many row blocks (an odd last one), chunks whose two blocks of a pair
see different numbers of pages, several splits, fp32 / fp16 / bf16 rows, against dequantize-then-attend.

Tolerance: that of the attention tests, against the rows that the cache holds."""
import numpy as np
import pytest

from oracle import tq_oracle as o
from tests.helpers import D, fill_cache, max_rel, stored_rows
from tests.test_gpu_attention import TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kf,vf", [("turbo3", "turbo3"), ("turbo4", "turbo4"), ("turbo4", "turbo2"), ("q8_0", "q8_0"), ("prod3", "turbo4")])
@pytest.mark.parametrize("group,chunk,lens", [(1, 128, [300, 128]), (1, 129, [129, 700]), (2, 128, [128, 257]), (8, 48, [40, 4100]),
                                              (4, 200, [1000, 200]), (8, 81, [81, 2000])])
def test_prefill_pairs(kf, vf, group, chunk, lens):
    import torch
    import turboquant_plus_b200 as tq
    rng = np.random.default_rng(chunk)
    hkv = 2
    cache = tq.PagedKVCache(D, hkv, num_pages=sum(-(-n // 128) for n in lens) + 1, k_format=kf, v_format=vf, seed=42)
    ks = [rng.standard_normal((n, hkv, D)).astype(np.float32) for n in lens]
    vs = [rng.standard_normal((n, hkv, D)).astype(np.float32) for n in lens]
    bt = fill_cache(cache, ks, vs, lens, rng)
    q = rng.standard_normal((len(lens), chunk, hkv * group, D)).astype(np.float32)
    qt, lt = torch.as_tensor(q).cuda(), torch.tensor(lens)
    out = cache.prefill_attend(qt, bt, lt)
    assert cache.kernel_status() == 0 and torch.equal(out, cache.prefill_attend(qt, bt, lt))
    for dt in (torch.float16, torch.bfloat16):                 # rows widened exactly, outputs rounded to nearest
        assert torch.equal(cache.prefill_attend(qt.to(dt), bt, lt), cache.prefill_attend(qt.to(dt).float(), bt, lt).to(dt))
    errs = []
    for b, n in enumerate(lens):
        pages = bt[b, :-(-n // 128)].numpy()
        kh, vh = (stored_rows(cache, w, pages, n).transpose(1, 0, 2)[None] for w in "kv")
        lo = max(0, chunk - n)
        some = np.unique(np.concatenate([[lo, chunk - 1], rng.integers(lo, chunk, 24)]))     # the oracle is slow
        got = out[b].cpu().numpy()
        assert not got[:lo].any()
        for i in some:
            m = n - chunk + i + 1
            ref = o.attend_gqa(q[b, i][None].astype(np.float64), kh[:, :, :m], vh[:, :, :m], [m])[0]
            errs.append(max_rel(got[i], ref))
    assert max(errs) < TOL, f"{kf}/{vf}: {max(errs)}"


def _coarse_bytes(chunk, hq, hkv, pages, sms):
    """The workspace of one sequence's chunk with at least eight pages a split, in the form that needs more."""
    blocks, most = -(-chunk * (hq // hkv) // 128), 0
    for cg in (1, 2):
        base, slots = -(-blocks // cg) * hkv, sms // cg
        s = min(range(1, min(max(pages // 8, 1), 64) + 1), key=lambda c: -(-base * c // slots) * (-(-pages // c) + 12))
        splits = -(-pages // -(-pages // s))
        total = blocks * hkv * splits * (128 * D * 4 + 128 * 2 * 4) + 65536 * 4 + 256
        most = max(most, -(-total // 256) * 256)
    return most


@pytest.mark.parametrize("kf,vf", [("turbo3", "turbo3"), ("q8_0", "turbo2"), ("prod3", "turbo3")])
@pytest.mark.parametrize("hq,hkv,pages", [(32, 8, 20), (16, 2, 40), (4, 1, 9)])
def test_workspaces_that_the_finest_plan_does_not_fit(kf, vf, hq, hkv, pages):
    """A workspace for fewer splits serves the call: sized for a prompt's largest chunk, it has to do for its last one."""
    import torch
    import turboquant_plus_b200 as tq
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    gen = torch.Generator(device="cuda").manual_seed(pages)
    cache = tq.PagedKVCache(D, hkv, pages, 128, kf, vf, seed=42)
    n = pages * 128 - 40
    cache.append(*(torch.randn((n, hkv, D), device="cuda", generator=gen) for _ in range(2)), torch.arange(n, device="cuda"))
    table, lens = torch.arange(pages, dtype=torch.int32)[None], torch.tensor([n])
    smaller = 0
    for chunk in (16, 26, 40, 64, 96, 130, 200, 320, 512):
        q = torch.randn((1, chunk, hq, D), device="cuda", generator=gen)
        size = _coarse_bytes(chunk, hq, hkv, pages, sms)
        smaller += size < tq._native.load().tq_prefill_workspace_bytes(1, chunk, hq, hkv, pages)
        ws = torch.zeros(size, dtype=torch.uint8, device="cuda")
        out, want = cache.prefill_attend(q, table, lens, workspace=ws), cache.prefill_attend(q, table, lens)
        assert cache.kernel_status(ws) == 0 and cache.kernel_status() == 0
        # (probabilities are fp16 numbers relative to the largest of their split: either side is within TOL of exact sums)
        assert float((out - want).abs().max() / want.abs().max()) < 2 * TOL
        if kf == "turbo3":
            with pytest.raises(RuntimeError):
                cache.prefill_attend(q, table, lens, workspace=torch.zeros(65536 * 4 + 256, dtype=torch.uint8, device="cuda"))
    assert smaller >= 3


@pytest.mark.parametrize("kf,vf", [("turbo3", "turbo3"), ("turbo4", "turbo2"), ("prod3", "turbo3")])
@pytest.mark.parametrize("hkv,group,chunk,lens", [(8, 2, 128, [128, 1]), (8, 4, 64, [64, 200]), (8, 4, 90, [700, 90])])
def test_first_page_beside_the_rows(kf, vf, hkv, group, chunk, lens):
    """Dense rotations, whose rows need more of the memory that the first page's keys are dequantized into meanwhile, rows of both widths,
    sequences of one page and of several: every query against a decode call of its own."""
    import torch
    import turboquant_plus_b200 as tq
    gen = torch.Generator(device="cuda").manual_seed(chunk)
    pages = -(-max(lens) // 128)
    n = len(lens) * pages * 128
    cache = tq.PagedKVCache(D, hkv, len(lens) * pages, 128, kf, vf, seed=42, rotation="dense")
    k, v = (torch.randn((n, hkv, D), device="cuda", generator=gen) for _ in range(2))
    cache.append(k, v, torch.arange(n, device="cuda"))
    bt = torch.randperm(len(lens) * pages, device="cuda", generator=gen).to(torch.int32).view(len(lens), pages)
    sl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    q = torch.randn((len(lens), chunk, hkv * group, D), device="cuda", generator=gen).half()
    got = cache.prefill_attend(q, bt, sl)
    assert cache.kernel_status() == 0 and torch.equal(got, cache.prefill_attend(q.float(), bt, sl).half())
    for i in range(0, chunk, 7):
        seen = (sl - chunk + 1 + i).clamp(min=0)
        live = (seen > 0).cpu()
        assert not got[:, i][~live].any()
        if live.any():
            want = cache.attend(q[:, i].contiguous(), bt, seen)
            assert max_rel(got[:, i][live].float().cpu().numpy(), want[live].float().cpu().numpy()) < 2e-3
