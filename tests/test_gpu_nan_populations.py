"""FP64 populations that are NaN -- a demographic change over areas without
people, whose shares are 0 / 0, or a start population that is NaN -- make
their rates NaN: the plain form gives the status the oracle gives."""
import numpy as np
import pytest

from beep_gb300 import capi, model_builder as mb, synth
from oracle_lib import oracle_simulate

pytestmark = pytest.mark.gpu


def outcome(run, b):
    try:
        run(b)
        return b.L.tolist(), b.pop.tolist()
    except (capi.BeepError, RuntimeError) as e:
        return next(n for n in capi.STATUS.values() if n in str(e))


def model(empty):
    w = synth.seir_hd_democat(seed=20261203, narea=6, nage=2, days=20)
    arr = dict(mb.model_arrays(w))
    if empty:
        pop = np.array(arr["pop_init"], copy=True)
        a0, a1 = np.asarray(arr["dcc_area_ptr"])[1:3]
        pop[np.asarray(arr["dcc_area"])[a0:a1]] = 0         # the second change's areas
        arr["pop_init"] = pop
    return capi.Model(arr), [capi.Tables(mb.param_tables_batch(w, [2.0], [4.0], [5.0])[0])]


@pytest.mark.parametrize("empty", (False, True))
def test_change_over_areas_without_people(empty):
    m, tabs = model(empty)
    assert m.pop64 and m.ndemocat_change == 2
    dm = capi.DeviceModel(m)
    b = lambda: capi.Batch(m, tabs, 3, 7, want_pop=True)    # noqa: E731
    got, want = outcome(dm.simulate, b()), outcome(lambda x: oracle_simulate(m, x), b())
    dm.close()
    if empty:
        assert want == "NAN_RATE" and got == want
    else:
        assert got[1] == want[1]


def test_start_populations_that_are_nan():
    m, tabs = model(False)
    pop = np.repeat(m.arr["pop_init"].reshape(1, m.narea, m.ncomp, m.ndemocatpos), 3, axis=0)
    pop[1, 2, 0, 1] = np.nan
    dm = capi.DeviceModel(m)
    b = lambda: capi.Batch(m, tabs, 3, 7, ti=4, pop_in=pop, want_pop=True)    # noqa: E731
    got, want = outcome(dm.simulate, b()), outcome(lambda x: oracle_simulate(m, x), b())
    dm.close()
    assert want == "NAN_RATE" and got == want
