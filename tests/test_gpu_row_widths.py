"""quantize_device on rows that are wider than the quantizer's dimension (a slice of the columns without a copy): the first d
columns count, as for a contiguous copy of them; narrower rows are refused."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rotation", ["wht", "dense"])
@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("kind", ["PolarQuant", "TurboQuant"])
def test_wider_and_narrower_rows(rotation, packed, kind):
    import torch
    import turboquant_plus_b200 as tq
    gen = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn((77, 192), device="cuda", generator=gen)
    quantizer = getattr(tq, kind)(128, 3, seed=1, rotation=rotation)
    got = quantizer.quantize_device(x, packed=packed, want_scale=True)
    want = quantizer.quantize_device(x[:, :128].contiguous(), packed=packed, want_scale=True)
    assert got.keys() == want.keys()
    for name in want:
        assert got[name].shape == want[name].shape and torch.equal(got[name], want[name]), name
    with pytest.raises(ValueError):
        quantizer.quantize_device(x[:, :96].contiguous(), packed=packed)
