"""The filter's resampling over the sizes its kernel splits on (part warps, one
and several passes of the CTA, arrays beyond shared memory) against the
oracle: ancestors identical, estimate to 1e-12 -- the plain form's bar."""
import numpy as np
import pytest

from beep_gb300 import capi
from golden_util import load
from oracle_lib import oracle_pf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", (1, 2, 31, 33, 257, 1024, 1025, 8192, 8193))
def test_resampling_sizes(N):
    b, m, tabs, seed = load("tiny_pf")
    dm = capi.DeviceModel(m)
    for invT in (1.0, 0.02):                   # few survivors, many survivors
        ll, lls, L, anc = dm.pf_loglik(tabs[0], N, seed + N, 5, invT, m.sections)
        llo, llso, Lo, anco = oracle_pf(m, tabs[0], N, seed + N, 5, invT, m.sections)
        assert np.array_equal(anc, anco)
        np.testing.assert_allclose(lls, llso, rtol=1e-12)
        np.testing.assert_allclose(L, Lo, rtol=1e-12)
        assert abs(ll - llo) <= 1e-12 * abs(llo)
    dm.close()
