"""The force of infection with four targets per quad of lanes (640-thread CTAs,
more than 320 areas, up to 12 ages, the matrix read from L2): area counts
divisible by four (float4 loads), even (float2) and odd (single loads, one to
three targets in the last quad), and an age stride of 4, 8 and 12.  Its sums
are those of the two-target form, which the 320-thread layouts run: counts and
populations equal bit for bit, in simulations and in chains; and short runs
follow the plain form."""
import numpy as np
import pytest

from beep_gb300 import capi, model_builder as mb, synth

pytestmark = pytest.mark.gpu

SIZES = [(321, 1), (322, 5), (323, 9), (324, 1), (324, 5), (353, 12), (356, 9), (357, 4)]


@pytest.fixture(params=SIZES, ids=lambda s: "%dx%d" % s)
def case(request):
    narea, nage = request.param
    w = synth.seir_hd_small(seed=20261001 + narea, narea=narea, nage=nage, days=6, steps_per_day=2)
    w.obs_kind = "hosp_pop"
    w.seed_E[:, :] = 6
    m = capi.Model(mb.model_arrays(w))
    rng = np.random.default_rng(narea)
    tabs = [[capi.Tables(t) for t in mb.param_tables_batch(w, *rng.uniform([2.2, 3.6, 4.5], [2.8, 4.4, 5.5], (6, 3)).T)]
            for _ in range(2)]
    capi.set_option("fast_foi", capi.FOI_SIMT)
    yield m, tabs
    capi.set_option("fast_foi", capi.FOI_AUTO)
    capi.set_option("fast_ctas_per_sm", 0)


def test_simulations(case):
    m, (tabs, _) = case
    dm = capi.DeviceModel(m)
    P = 12
    kw = dict(group_of=np.arange(P) % 6, want_pop=True, want_transnum=True)
    out = {}
    for ctas in (1, 2):
        capi.set_option("fast_ctas_per_sm", ctas)
        db = capi.DeviceBatch(dm, capi.Batch(m, tabs, P, 4, form=capi.FORM_FAST, **kw))
        assert (db.foi_path(), db.ctas_per_sm()) == (1, ctas)
        out[ctas] = db.run()
        db.close()
    assert np.array_equal(out[1].transnum, out[2].transnum) and np.array_equal(out[1].pop, out[2].pop)
    np.testing.assert_allclose(out[1].L, out[2].L, rtol=1e-6)
    p = dm.simulate(capi.Batch(m, tabs, P, 4, **kw))
    same = np.array([np.array_equal(p.transnum[k], out[1].transnum[k]) for k in range(P)])
    assert same.mean() >= 0.4
    np.testing.assert_allclose(out[1].L[same], p.L[same], rtol=1e-6)
    dm.close()


def test_chains(case):
    m, (t0, t1) = case
    dm = capi.DeviceModel(m)
    nc = 6
    go, so = np.arange(nc), np.arange(nc, dtype=np.uint32)
    out = {}
    for ctas in (1, 2):
        capi.set_option("fast_ctas_per_sm", ctas)
        ch = capi.MbpChains(dm, nc, form=capi.FORM_FAST)
        ch.initialise(t0, 9, group_of=go, stream_of=so)
        a = [ch.read_state(k)[0] for k in range(nc)]
        L = ch.propose(t1, 9, group_of=go, stream_of=so + 100)
        assert ch.ctas_per_sm() == ctas
        ch.accept(np.ones(nc, np.uint8))
        out[ctas] = (a, [ch.read_state(k)[0] for k in range(nc)], L)
        ch.close()
    for i in (0, 1):
        assert all(np.array_equal(x, y) for x, y in zip(out[1][i], out[2][i]))
    np.testing.assert_allclose(out[1][2], out[2][2], rtol=1e-6)
    dm.close()
