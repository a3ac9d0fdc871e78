"""The dense kernels' shared-memory limit with several host threads: the limit of a kernel belongs to the process, and a call
of a smaller dimension on another thread must not lower it under a thread that has raised it."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large,small", [(256, 136), (128, 40)])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_smaller_dimension_on_another_thread(large, small, dtype):
    import torch
    import turboquant_plus_b200 as tq
    n = 20000                                      # tiles of 64 vectors up to d = 128, of 32 above
    gen = torch.Generator(device="cuda").manual_seed(1)
    x = {d: torch.randn((n, d), device="cuda", generator=gen, dtype=getattr(torch, dtype)) for d in (large, small)}
    quantizers = {d: tq.TurboQuant(d, 3, seed=1) for d in x}
    want, failed = {}, []

    def call(d):
        try:
            code = quantizers[d].quantize(x[d])
            got = torch.cat([code.mse_indices.double(), quantizers[d].dequantize(code).double()], dim=1)
            torch.cuda.synchronize()
            if not torch.equal(want.setdefault(d, got), got):
                failed.append("other results")
        except Exception as e:                     # an assertion of a thread does not reach pytest
            failed.append(e)

    call(large)
    other = threading.Thread(target=call, args=(small,))
    other.start()
    other.join()
    call(large)
    assert not failed, failed
