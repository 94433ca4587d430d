"""The plain form's draws, decided in FP32 where a bound allows and in FP64
otherwise (rng_filter.cuh), are the FP64 samplers' integers: trajectories equal
to the oracle's at populations from a few people (means below 1, inversion
only) to 1e9 (means of 1e7, where the bounds send draws back to FP64)."""
import numpy as np
import pytest

from beep_gb300 import capi, model_builder as mb, synth
from oracle_lib import oracle_mbp, oracle_simulate

pytestmark = pytest.mark.gpu


def model(people, seeded):
    """5 areas x 3 ages over 40 days, `people` per area and age, `seeded` of them exposed."""
    w = synth.seir_hd_small(seed=20260201, narea=5, nage=3, days=40, steps_per_day=2)
    w.pop = np.full((5, 3), people, np.int64)
    w.seed_E = np.full((5, 3), seeded, np.int64)
    return w, capi.Model(mb.model_arrays(w))


@pytest.mark.parametrize("people, seeded", [(4, 2), (60, 30), (2000, 400), (10**6, 10**5), (10**8, 10**7)])
def test_filtered_draws_are_the_fp64_draws(people, seeded):
    w, m = model(people, seeded)
    rng = np.random.default_rng(people)
    tabs = [capi.Tables(t) for t in mb.param_tables_batch(w, *synth.abc_smc_priors(rng, 4))]
    P = 40
    go = np.arange(P) % 4
    dm = capi.DeviceModel(m)
    g = dm.simulate(capi.Batch(m, tabs, P, 77, group_of=go, want_transnum=True, want_pop=True))
    o = oracle_simulate(m, capi.Batch(m, tabs, P, 77, group_of=go, want_transnum=True, want_pop=True))
    assert np.array_equal(g.transnum, o.transnum)
    assert np.array_equal(g.pop, o.pop)
    nc = 16
    gi, gp = np.arange(nc) % 4, (np.arange(nc) + 1) % 4
    si, sp = np.arange(nc, dtype=np.uint32), np.arange(nc, dtype=np.uint32) + 500
    ref = oracle_mbp(m, tabs, gi, gp, 77, si, sp, capi.INF_DIF_UPDATE, None, want_tn=True)
    ch = capi.MbpChains(dm, nc)
    ch.initialise(tabs, 77, group_of=gi, stream_of=si)
    ch.propose(tabs, 77, group_of=gp, stream_of=sp)
    ch.accept(np.ones(nc, np.uint8))
    for k in range(nc):
        assert np.array_equal(ch.read_state(k)[0], ref["tn_prop"][k])
    ch.close()
    dm.close()


@pytest.mark.parametrize("infectivity, people, zero_entry", [(1.0, 2000, False), (3.0, 2000, False), (0.37, 2000, False),
                                                              (2048.0, 2000, False), (1024.0, 10**8, False),
                                                              (1.0, 2000, True)])
def test_area_mixing_sums_are_the_fp64_sums(infectivity, people, zero_entry):
    """The infectious counts' products with the mixing matrix on the integer pipe (integer
    infectivities up to 1024, sums below 2^32, a matrix of ordinary values) and on the FP64 pipe
    (otherwise): trajectories and chain states equal to the oracle's."""
    w, _ = model(people, people // 10)
    arr = mb.model_arrays(w)
    if zero_entry:
        arr["M_val"] = arr["M_val"].copy()
        arr["M_val"][1] = 0.0
    m = capi.Model(arr)
    raw = mb.param_tables_batch(w, *synth.abc_smc_priors(np.random.default_rng(5), 3))
    tabs = []
    for t in raw:
        inf = t["infectivity"].copy()
        inf[2] = infectivity
        tabs.append(capi.Tables(dict(t, infectivity=inf, beta_rows=t["beta_rows"] / infectivity)))
    P = 24
    go = np.arange(P) % 3
    dm = capi.DeviceModel(m)
    g = dm.simulate(capi.Batch(m, tabs, P, 78, group_of=go, want_transnum=True, want_pop=True))
    o = oracle_simulate(m, capi.Batch(m, tabs, P, 78, group_of=go, want_transnum=True, want_pop=True))
    assert np.array_equal(g.transnum, o.transnum) and np.array_equal(g.pop, o.pop)
    nc = 9
    gi, gp = np.arange(nc) % 3, (np.arange(nc) + 1) % 3
    si, sp = np.arange(nc, dtype=np.uint32), np.arange(nc, dtype=np.uint32) + 500
    for iu in (capi.INF_DIF_UPDATE, capi.INF_UPDATE):
        ref = oracle_mbp(m, tabs, gi, gp, 78, si, sp, iu, None, want_tn=True)
        ch = capi.MbpChains(dm, nc)
        ch.initialise(tabs, 78, group_of=gi, stream_of=si)
        np.testing.assert_allclose(ch.state_likelihood(tabs, group_of=gp), ref["Li_fixed"], rtol=1e-12)
        ch.propose(tabs, 78, group_of=gp, stream_of=sp, inf_update=iu)
        ch.accept(np.ones(nc, np.uint8))
        for k in range(nc):
            assert np.array_equal(ch.read_state(k)[0], ref["tn_prop"][k])
        ch.close()
    dm.close()
