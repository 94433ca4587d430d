"""A proposal from a state whose means are NaN (rates that were refused with
NAN_RATE, accepted all the same): a cell with a NaN current mean and a finite
proposed one is the binomial of a NaN probability, 0, in both forms."""
import numpy as np
import pytest

from beep_gb300 import capi, model_builder as mb, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", (capi.FORM_PLAIN_FP64, capi.FORM_FAST))
def test_counts_under_nan_means_are_zero(form):
    w = synth.seir_hd_small(seed=20260902, narea=7, nage=2, days=20, steps_per_day=2)
    w.obs_kind = "hosp_pop"
    w.seed_E[:, :] = 200
    m = capi.Model(mb.model_arrays(w))
    raw = mb.param_tables_batch(w, [2.5], [4.0], [5.0])[0]
    bad_rate = raw["transrate"].copy()
    bad_rate[1] = np.nan                                   # E -> I
    good, bad = capi.Tables(raw), capi.Tables(dict(raw, transrate=bad_rate))
    dm = capi.DeviceModel(m)
    ch = capi.MbpChains(dm, 3, form=form)
    ch.initialise([good], 5)
    tn = np.stack([ch.read_state(k)[0] for k in range(3)])
    with pytest.raises(capi.BeepError) as e:
        ch.set_state([bad], tn)
    assert e.value.status == 2                             # BEEP_NAN_RATE
    ch.accept(np.ones(3, np.uint8))
    old = [ch.read_state(k) for k in range(3)]
    ch.propose([good], 6, stream_of=np.arange(3, dtype=np.uint32) + 50)
    ch.accept(np.ones(3, np.uint8))
    for k in range(3):
        n0, mean0 = old[k]
        n1, mean1 = ch.read_state(k)
        cells = np.isnan(mean0) & (mean1 > 0)
        assert (n0[cells] > 0).any()
        assert not n1[cells].any()
    ch.close()
    dm.close()
