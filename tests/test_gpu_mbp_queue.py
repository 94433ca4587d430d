"""Fast chains whose proposals queue their draws, over column counts around the
32-column groups and the CTA sizes, odd area counts of the four-target force of
infection, SIMU masks and one chain that gives up: against the plain chains on
the same streams, with the bars of the fast-form chain test (at least 40% of
the proposals identical; L within 1e-6 where they are)."""
import numpy as np
import pytest

from beep_gb300 import capi, model_builder as mb, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("masked", (False, True))
@pytest.mark.parametrize("narea, nage", [(1, 1), (31, 1), (33, 1), (16, 2), (43, 3), (129, 1), (131, 5), (150, 9), (202, 4)])
def test_queued_proposals_follow_the_plain_chains(narea, nage, masked):
    w = synth.seir_hd_small(seed=20260400 + narea, narea=narea, nage=nage, days=25, steps_per_day=2)
    w.obs_kind = "hosp_pop"
    w.seed_E[:, :] = 6
    m = capi.Model(mb.model_arrays(w))
    rng = np.random.default_rng(narea)
    nc = 24
    th = np.stack([rng.uniform(2.2, 2.8, nc), rng.uniform(3.6, 4.4, nc), rng.uniform(4.5, 5.5, nc)], 1)
    t0 = [capi.Tables(t) for t in mb.param_tables_batch(w, *th.T)]
    t1 = [capi.Tables(t) for t in mb.param_tables_batch(w, *(th * np.exp(rng.normal(0, 0.05, th.shape))).T)]
    simu = (rng.random((nc, m.ndivision, m.narea)) < 0.2).astype(np.uint8) if masked else None
    dm = capi.DeviceModel(m)
    go, so = np.arange(nc), np.arange(nc, dtype=np.uint32)
    start = capi.MbpChains(dm, nc)
    start.initialise(t0, 9, group_of=go, stream_of=so)
    tn0 = np.stack([start.read_state(k)[0] for k in range(nc)])
    out = {}
    for form in (capi.FORM_PLAIN_FP64, capi.FORM_FAST):
        ch = capi.MbpChains(dm, nc, form=form)
        ch.set_state(t0, tn0, group_of=go)               # the same start in both forms
        L = ch.propose(t1, 9, group_of=go, stream_of=so + 100, simu=simu)
        ch.accept(np.ones(nc, np.uint8))
        out[form] = (L, [ch.read_state(k)[0] for k in range(nc)])
        ch.close()
    start.close()
    (Lp, tp), (Lf, tf) = out[capi.FORM_PLAIN_FP64], out[capi.FORM_FAST]
    same = np.array([np.array_equal(a, b) for a, b in zip(tp, tf)])
    assert same.mean() >= 0.4
    np.testing.assert_allclose(Lf[same], Lp[same], rtol=1e-6)
    dm.close()


def test_a_queued_draw_that_gives_up_is_a_timeout():
    w = synth.seir_hd_small(seed=20260411, narea=40, nage=3, days=30, steps_per_day=2)
    w.seed_E[:, :] = 2000                                # means far above 10: rejection samplers
    m = capi.Model(mb.model_arrays(w))
    tabs = [capi.Tables(t) for t in mb.param_tables_batch(w, [2.5, 2.0], [4.0, 4.4], [5.0, 5.5])]
    dm = capi.DeviceModel(m)
    ch = capi.MbpChains(dm, 4, form=capi.FORM_FAST)
    ch.initialise([tabs[0]], 3)
    L = ch.propose([tabs[1]], 3, stream_of=np.arange(4) + 10)
    capi.set_option("sampler_iteration_limit", 1)
    try:
        with pytest.raises(capi.BeepError) as e:
            ch.propose([tabs[1]], 3, stream_of=np.arange(4) + 10)
        assert e.value.status == 4                       # BEEP_TIMEOUT
    finally:
        capi.set_option("sampler_iteration_limit", 0)
    assert np.array_equal(ch.propose([tabs[1]], 3, stream_of=np.arange(4) + 10), L)
    ch.close()
    dm.close()
