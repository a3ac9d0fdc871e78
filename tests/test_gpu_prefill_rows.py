"""Short chunks over q8_0 and PROD tensors, on both sides of the size at which they go from rows of the decode kernel to tiles:
every query against a decode call of its own, chunks longer than their sequence (the first queries see nothing), rows of 16
bits, output and workspace given.

Tolerance: that of the attention tests."""
import pytest

from tests.helpers import max_rel

pytestmark = pytest.mark.gpu
D = 128


@pytest.mark.parametrize("kf,vf,rotation", [("q8_0", "turbo2", "wht"), ("q8_0", "q8_0", "wht"), ("prod3", "turbo3", "wht"),
                                            ("prod4", "turbo4", "wht"), ("prod3", "turbo3", "dense")])
@pytest.mark.parametrize("hkv,group,lens,chunk", [(2, 4, [1], 1), (8, 4, [4000], 1), (8, 4, [4000, 3], 6), (2, 8, [300, 129, 5], 8),
                                                  (1, 4, [9000], 20), (8, 8, [2000], 12), (1, 16, [500], 4), (8, 4, [700, 40], 40)])
def test_short_chunks(kf, vf, rotation, hkv, group, lens, chunk):
    import torch
    import turboquant_plus_b200 as tq
    gen = torch.Generator(device="cuda").manual_seed(chunk)
    pages = -(-max(lens) // 128)
    cache = tq.PagedKVCache(D, hkv, len(lens) * pages, 128, kf, vf, seed=42, rotation=rotation)
    n = len(lens) * pages * 128
    k, v = (torch.randn((n, hkv, D), device="cuda", generator=gen).half() for _ in range(2))
    cache.append(k, v, torch.arange(n, device="cuda"))
    bt = torch.randperm(len(lens) * pages, device="cuda", generator=gen).to(torch.int32).view(len(lens), pages)
    sl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    q = torch.randn((len(lens), chunk, hkv * group, D), device="cuda", generator=gen).half()
    got = cache.prefill_attend(q, bt, sl)
    assert cache.kernel_status() == 0 and torch.equal(got, cache.prefill_attend(q, bt, sl))
    if group <= 8:                                              # the decode kernel's range of heads
        for i in range(chunk):
            seen = (sl - chunk + 1 + i).clamp(min=0)
            want, live = cache.attend(q[:, i].contiguous(), bt, seen), (seen > 0).cpu()
            assert not got[:, i][~live].any()
            if live.any():
                assert max_rel(got[:, i][live].float().cpu().numpy(), want[live].float().cpu().numpy()) < 2e-3
    wide = cache.prefill_attend(q.float(), bt, sl)
    assert torch.equal(wide.half(), got)                        # rows widened exactly, outputs rounded to nearest
    from turboquant_plus_b200 import _native as nv
    need = nv.host().workspace_bytes(len(lens), hkv * group, hkv, pages, chunk)
    out, ws = torch.empty_like(q), torch.zeros(need, dtype=torch.uint8, device="cuda")
    assert cache.prefill_attend(q, bt, sl, out=out, workspace=ws) is out and torch.equal(out, got)
