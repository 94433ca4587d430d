"""NaN rates of the plain form: from a population size that is no divisor, with
and without external infections, on chip and off it, the status the oracle
gives."""
import numpy as np
import pytest

from beep_gb300 import capi, model_builder as mb, synth
from oracle_lib import oracle_simulate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("popsize", (0.0, float("nan"), float("inf"), -5.0))
@pytest.mark.parametrize("efoi", (0.0, 3.0))
@pytest.mark.parametrize("narea", (6, 2600))               # the step's tables in shared memory, or too many
def test_population_size_of_no_use(popsize, efoi, narea):
    w = synth.seir_hd_small(seed=20260901, narea=6, nage=1, days=4, steps_per_day=2)
    w.efoi = efoi
    arr = dict(mb.model_arrays(w), popsize=np.array([popsize]))
    t = dict(mb.param_tables_batch(w, [2.5], [4.0], [5.0])[0])
    if narea > 6:                                          # the same six areas over and over, without mixing
        rep = lambda x, ax: np.take(np.asarray(x), np.arange(narea) % 6, axis=ax)   # noqa: E731
        dims = np.asarray(arr["dims"]).copy()
        dims[0] = narea
        arr.update(dims=dims, M_diag=rep(arr["M_diag"], 0), M_factor=rep(arr["M_factor"], 0),
                   M_rowptr=np.zeros(narea + 1, np.int32), M_to=np.zeros(0, np.int32), M_val=np.zeros(0),
                   pop_init=rep(arr["pop_init"], 0))
        t.update(beta_row_of=rep(t["beta_row_of"], 1), areafactor=rep(t["areafactor"], 1), efoi_ref=rep(t["efoi_ref"], 1))
    m, tab = capi.Model(arr), capi.Tables(t)

    def outcome(run):
        b = capi.Batch(m, [tab], 3, 7, want_pop=True)
        try:
            run(b)
            return b.L.tolist(), b.pop.tolist()
        except (capi.BeepError, RuntimeError) as e:
            return next(n for n in capi.STATUS.values() if n in str(e))

    dm = capi.DeviceModel(m)
    got, want = outcome(dm.simulate), outcome(lambda b: oracle_simulate(m, b))
    dm.close()
    if isinstance(want, str):
        assert got == want
    else:
        assert got[1] == want[1]
        np.testing.assert_allclose(got[0], want[0], rtol=1e-12)
    if popsize != popsize or (popsize == 0.0 and efoi == 0.0):
        assert want == "NAN_RATE"
