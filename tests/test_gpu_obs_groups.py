"""Step-synchronous batches large enough for the observation kernel's four
particles per CTA, of sizes that leave one to three in the last: every
particle's log-likelihood and populations are those of a small batch (one
particle per CTA) on the same streams, bit for bit."""
import numpy as np
import pytest

from beep_gb300 import capi, model_builder as mb, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", (2432, 2433, 2434, 2435))
@pytest.mark.parametrize("obs_kind", ("cases_deaths", "hosp_pop", "obs_models"))
def test_large_batches_score_as_small_ones(P, obs_kind):
    w = synth.seir_hd_small(seed=20260501, narea=66, nage=2, days=20, steps_per_day=2)
    w.obs_kind = obs_kind
    w.seed_E[:, :] = 20
    m = capi.Model(mb.model_arrays(w))
    tabs = [capi.Tables(t) for t in mb.param_tables_batch(w, *synth.abc_smc_priors(np.random.default_rng(2), 3))]
    dm = capi.DeviceModel(m)
    capi.set_option("fast_foi", capi.FOI_BATCHED)
    try:
        big = dm.simulate(capi.Batch(m, tabs, P, 5, group_of=np.arange(P) % 3, want_pop=True, form=capi.FORM_FAST))
        pick = np.array([0, 1, 2, 3, 1000, P - 4, P - 3, P - 2, P - 1])
        few = dm.simulate(capi.Batch(m, tabs, len(pick), 5, group_of=pick % 3, stream_of=pick, want_pop=True,
                                     form=capi.FORM_FAST))
    finally:
        capi.set_option("fast_foi", capi.FOI_AUTO)
    assert np.array_equal(big.pop[pick], few.pop)
    assert np.array_equal(big.L[pick], few.L)
    dm.close()
