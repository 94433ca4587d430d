"""ABC-SMC weights over the shapes the kernel splits on (parameters per
instantiation and beyond, tiles and groups with remainders, one particle),
with previous weights of zero, new particles far from all previous ones (the
FP64 pass) and a form that is not positive definite, against the FP64 oracle.
Tolerance: the FP32 rounding of a quadratic form of up to 20 (2e-6 of its
half) plus that of the exponential, below 1e-5 as for the full-size test."""
import numpy as np
import pytest

from beep_gb300 import capi
from oracle_lib import oracle_abcsmc_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("definite", (True, False))
@pytest.mark.parametrize("nvar, nnew, nlast", [(1, 1, 1), (2, 33, 255), (3, 64, 8), (4, 31, 257), (5, 70, 519),
                                               (6, 95, 256), (7, 100, 263), (8, 40, 700), (16, 20, 90)])
def test_weights_over_shapes(nvar, nnew, nlast, definite):
    rng = np.random.default_rng(100 * nvar + nlast)
    tl = rng.uniform(-1, 1, (nlast, nvar))
    wl = rng.uniform(0.2, 2.0, nlast)
    wl[1::5] = 0.0
    tn = tl[rng.integers(0, nlast, nnew)] + rng.normal(0, 0.1, (nnew, nvar))
    tn[1::7] += 8.0 if definite else 0.0                   # far: the FP64 pass
    ic = np.eye(nvar) * rng.uniform(1.0, 3.0, nvar)
    if not definite:
        ic[0, 0] = -0.5
    lp = rng.normal(0, 0.3, nnew)
    g = capi.abcsmc_weights(tn, lp, tl, wl, ic, 1.2, normalise=False)
    o = oracle_abcsmc_weights(tn, lp, tl, wl, ic, 1.2, normalise=False)
    np.testing.assert_allclose(g, o, rtol=1e-5)
