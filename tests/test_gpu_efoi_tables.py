"""Batches, filters and chains kept across calls whose tables later come with
another number of external-force tables than the shared-memory layout was made
for (more, fewer, back again): equal to those of a fresh model on the same
tables, bit for bit."""
import numpy as np
import pytest

from beep_gb300 import capi, model_builder as mb, synth

pytestmark = pytest.mark.gpu

NAREA, NAGE = 9, 3


def workload():
    w = synth.seir_hd_small(seed=20260601, narea=NAREA, nage=NAGE, days=28, steps_per_day=2)
    w.obs_kind = "hosp_pop"
    return w, capi.Model(mb.model_arrays(w))


def tables(w, nefoi, R0=2.5):
    """One parameter set with `nefoi` external-force tables, each with its own age distribution."""
    t = mb.param_tables_batch(w, [R0], [4.0], [5.0])[0]
    S = t["efoi_spline"].shape[1]
    rng = np.random.default_rng(nefoi)
    return capi.Tables(dict(t, efoi_spline=np.outer(np.linspace(3.0, 30.0, nefoi), np.ones(S)),
                            efoi_agedist=rng.dirichlet(np.ones(NAGE), nefoi),
                            efoi_ref=(np.arange(NAREA) % nefoi).astype(np.int32).reshape(1, NAREA)))


ORDER = (1, 3, 2, 1, 7)


@pytest.mark.parametrize("N", (64, 1200))              # draws per (transition, column); per column
def test_filter_follows_the_number_of_tables(N):
    w, m = workload()
    dm = capi.DeviceModel(m)
    sections = [(0, 28), (28, 56)]
    for k, n in enumerate(ORDER):
        fresh = capi.DeviceModel(m)
        want = fresh.pf_loglik(tables(w, n), N, 40 + k, 5, 0.3, sections, form=capi.FORM_FAST)
        fresh.close()
        got = dm.pf_loglik(tables(w, n), N, 40 + k, 5, 0.3, sections, form=capi.FORM_FAST)
        assert got[0] == want[0] and all(np.array_equal(a, b) for a, b in zip(got[1:], want[1:]))
    dm.close()


@pytest.mark.parametrize("graph", (False, True))
def test_batch_follows_the_number_of_tables(graph):
    w, m = workload()
    dm = capi.DeviceModel(m)
    bt = capi.Batch(m, [tables(w, 1)], 200, 7, want_pop=True, form=capi.FORM_FAST)
    db = capi.DeviceBatch(dm, bt)
    for n in ORDER:
        t = tables(w, n)
        bt.groups[0] = t.st
        if graph:
            db.run_graph()
        else:
            db.stage()
            db.run()
        want = dm.simulate(capi.Batch(m, [t], 200, 7, want_pop=True, form=capi.FORM_FAST))
        assert np.array_equal(bt.L, want.L) and np.array_equal(bt.pop, want.pop)
    db.close()
    dm.close()


def test_chains_follow_the_number_of_tables():
    w, m = workload()
    dm = capi.DeviceModel(m)
    nc = 8
    so = np.arange(nc, dtype=np.uint32)

    def sweep(ch, n):
        ch.initialise([tables(w, n)], 9, stream_of=so)
        return ch.propose([tables(w, n, 2.7)], 9, stream_of=so + 100)

    ch = capi.MbpChains(dm, nc, form=capi.FORM_FAST)
    for n in ORDER:
        got = sweep(ch, n)
        ch.accept(np.ones(nc, np.uint8))
        fresh = capi.MbpChains(dm, nc, form=capi.FORM_FAST)
        want = sweep(fresh, n)
        fresh.accept(np.ones(nc, np.uint8))
        assert np.array_equal(got, want)
        for k in range(nc):
            assert np.array_equal(ch.read_state(k)[0], fresh.read_state(k)[0])
        fresh.close()
    ch.close()
    dm.close()


def test_graph_follows_the_sampler_limit():
    w, m = workload()
    w.seed_E[:, :] = 2000                              # rejection samplers
    m = capi.Model(mb.model_arrays(w))
    dm = capi.DeviceModel(m)
    bt = capi.Batch(m, [tables(w, 1)], 8, 7, form=capi.FORM_FAST)
    db = capi.DeviceBatch(dm, bt)
    db.run_graph()
    L = bt.L.copy()
    capi.set_option("sampler_iteration_limit", 1)
    try:
        with pytest.raises(capi.BeepError) as e:
            db.run_graph()
        assert e.value.status == 4                     # BEEP_TIMEOUT
    finally:
        capi.set_option("sampler_iteration_limit", 0)
    db.run_graph()
    assert np.array_equal(bt.L, L)
    db.close()
    dm.close()
