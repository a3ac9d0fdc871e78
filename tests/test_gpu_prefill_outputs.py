"""Chunked prefill over q8_0 and PROD tensors into every kind of ``out`` that a copy can fill (strided, of another type, not
aligned, on the host), and with workspaces of other calls: the values are those of the plain call."""
import pytest

pytestmark = pytest.mark.gpu
D = 128


@pytest.mark.parametrize("kf,vf", [("q8_0", "turbo2"), ("prod3", "turbo3")])
def test_outputs_and_workspaces(kf, vf):
    import torch
    import turboquant_plus_b200 as tq
    gen = torch.Generator(device="cuda").manual_seed(1)
    cache = tq.PagedKVCache(D, 2, 4, 128, kf, vf, seed=42)
    rows = [torch.randn((300, 2, D), device="cuda", generator=gen).half() for _ in range(2)]
    cache.append(*rows, torch.arange(300, device="cuda"))
    q = torch.randn((1, 40, 8, D), device="cuda", generator=gen).half()
    bt, lens = torch.arange(3, device="cuda", dtype=torch.int32)[None], torch.tensor([300], device="cuda", dtype=torch.int32)
    want = cache.prefill_attend(q, bt, lens)
    wide = torch.full((1, 40, 8, 2 * D), 7.0, device="cuda", dtype=torch.float16)
    turned = torch.full((1, 8, 40, D), 7.0, device="cuda", dtype=torch.float16)
    shifted = torch.full((want.numel() + 8,), 7.0, device="cuda", dtype=torch.float16)
    for out in (wide[..., :D], turned.transpose(1, 2), shifted[1:1 + want.numel()].view(want.shape),
                torch.empty_like(want, dtype=torch.float64), torch.empty_like(want, device="cpu")):
        got = cache.prefill_attend(q, bt, lens, out=out)
        assert got is out and torch.equal(out.to(want), want)
    assert (wide[..., D:] == 7.0).all() and shifted[0] == 7.0 and (shifted[1 + want.numel():] == 7.0).all()
    for workspace in (torch.zeros(256, dtype=torch.uint8, device="cuda"), cache.workspace(1, 8, 3)):
        assert torch.equal(cache.prefill_attend(q, bt, lens, workspace=workspace), want)
