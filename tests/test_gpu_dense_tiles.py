"""The fp64 tensor-core kernels of the dense mode at the edges of their tiles (16, 32 or 64 vectors, 16 or 32 outputs
per warp, k-steps of 8, d up to 256; wider vectors take the kernel beside them), against the oracle.

Tolerance: indices and signs equal except where the fp64 value lies within 1e-12 (fp64 inputs) of a boundary (the sums are fp64 in
another order: d eps ~ 3e-14 of the largest term); norms 1e-6 relative (fp32); reconstructions 1e-6 (fp32 norms)."""
import numpy as np
import pytest

from oracle import tq_oracle as o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n", [(1, 5), (7, 33), (8, 1), (31, 64), (64, 65), (100, 31), (128, 97), (128, 15), (130, 40), (200, 33),
                                 (255, 17), (256, 64), (264, 9), (96, 9700), (128, 4737), (128, 9473)])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_dense_tiles(d, n, dtype):
    import turboquant_plus_b200 as tq
    rng = np.random.default_rng(d + n)
    x = (rng.standard_normal((n, d)) * np.exp(0.5 * rng.standard_normal((n, 1)))).astype(dtype)
    x[n // 2] = 0.0
    t = tq.TurboQuant(d, 3, seed=5)
    rot, cent, s = t.polar_quant.rotation, t.polar_quant.centroids, t.qjl.S
    code = t.quantize(x)
    ref = o.prod_quantize(x, rot, cent, s, 3)
    idx, nrm, y = o.polar_quantize(x, rot, cent, return_rotated=True)
    gap = np.abs(y[..., None] - (cent[1:] + cent[:-1]) / 2).min(axis=-1)
    # fp32 inputs: the norm is an fp32 sum whose order NumPy's SIMD build does not keep, up to 2 ulp (2.4e-7) off, and the
    # division by it rounds at 6e-8; both scale y
    assert (code.mse_indices == idx)[gap > (1e-12 if dtype == "float64" else 3e-7 * np.abs(y))].all()
    coded = (code.mse_indices == idx).all(axis=1)     # a vector with another index has another residual
    assert coded.mean() > 0.99
    live = (nrm > 0) & coded
    assert np.allclose(code.vector_norms, nrm, rtol=1e-6, atol=0)
    # with fp32 norms in the residual, a projection below the norm's rounding may take either sign
    _, _, res = o.polar_residual(x, rot, cent)
    p = res @ s.T
    sure = (np.abs(p) > 4e-7 * nrm[:, None] * np.sqrt(d)) & coded[:, None]
    assert (code.qjl_signs == ref.qjl_signs)[sure].all()
    assert np.allclose(code.residual_norms[live], ref.residual_norms[live], rtol=1e-5, atol=1e-6 * nrm.max())
    back, want = t.dequantize(code), o.prod_dequantize(ref, rot, cent, s)
    same = (code.qjl_signs == ref.qjl_signs).all(axis=1) & coded
    # (d = 1: the corrected code reproduces x, the residual is rounding noise and its signs are anything)
    assert same.mean() > 0.9 or d == 1
    assert np.abs((back - want) * same[:, None]).max() <= 1e-6 * max(np.abs(want).max(), 1e-30)
    # column slices: the outlier quantizer writes and accumulates into parts of wider rows
    if d >= 8:
        oq = tq.OutlierTurboQuant(d, 2.5, seed=3)
        oc = oq.quantize(x)
        i0, n0 = o.polar_quantize(x[:, :oq.n_outlier], oq.pq_outlier.rotation, oq.pq_outlier.centroids)
        assert (oc.outlier_indices == i0).mean() > 1 - 1e-4 and np.allclose(oc.outlier_norms, n0, rtol=1e-6)
        assert np.isfinite(oq.dequantize(oc)).all()
