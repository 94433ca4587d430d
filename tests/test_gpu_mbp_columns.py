"""Proposals that queue their draws against those that draw column by column,
count for count.  The queue needs room beside the chain's state: with three
or four chains per SM there is none (one 640-thread CTA per SM has it), nor for small
models whose observation slots nearly fill the shared memory."""
import numpy as np
import pytest

from beep_gb300 import capi, model_builder as mb, synth

pytestmark = pytest.mark.gpu


def workload(narea, nage, seed_E):
    w = synth.seir_hd_small(seed=20261100 + narea, narea=narea, nage=nage, days=25, steps_per_day=2)
    w.obs_kind = "hosp_pop"
    w.seed_E[:, :] = seed_E
    rng = np.random.default_rng(narea)
    th = rng.uniform([2.2, 3.6, 4.5], [2.8, 4.4, 5.5], (8, 3))
    th1 = th * np.exp(rng.normal(0, 0.2, th.shape))
    return mb.model_arrays(w), [[capi.Tables(t) for t in mb.param_tables_batch(w, *x.T)] for x in (th, th1)]


def proposals(arr, tabs, masked):
    m = capi.Model(arr)
    nc = 16
    go, so = np.arange(nc) % 8, np.arange(nc, dtype=np.uint32)
    simu = (np.random.default_rng(3).random((nc, m.ndivision, m.narea)) < 0.2).astype(np.uint8) if masked else None
    dm = capi.DeviceModel(m)
    ch = capi.MbpChains(dm, nc, form=capi.FORM_FAST)
    ch.initialise(tabs[0], 9, group_of=go, stream_of=so)
    out = []
    for k in (1, 0, 1):                                    # up, down and up again in mean
        L = ch.propose(tabs[k], 9, group_of=go, stream_of=so + 100 * (len(out) + 1), simu=simu)
        ch.accept(np.ones(nc, np.uint8))
        out.append(([ch.read_state(c) for c in range(nc)], L))
    per_sm = ch.ctas_per_sm()
    ch.close()
    dm.close()
    return out, per_sm


def equal(a, b):
    for (sa, La), (sb, Lb) in zip(a, b):
        for (na, ma), (nb, mb_) in zip(sa, sb):
            assert np.array_equal(na, nb) and np.array_equal(ma, mb_)
        np.testing.assert_allclose(La, Lb, rtol=1e-6)


@pytest.mark.parametrize("masked", (False, True))
@pytest.mark.parametrize("narea, nage, seed_E", [(257, 1, 6), (70, 4, 200), (65, 5, 6), (129, 2, 2000), (97, 7, 40), (230, 3, 6)])
def test_one_and_several_chains_per_sm(narea, nage, seed_E, masked):
    arr, tabs = workload(narea, nage, seed_E)
    out = {}
    for k in (1, 4):
        capi.set_option("fast_ctas_per_sm", k)
        try:
            out[k], per_sm = proposals(arr, tabs, masked)
        finally:
            capi.set_option("fast_ctas_per_sm", 0)
        assert per_sm == 1 if k == 1 else per_sm >= 3       # (three where four do not fit: no room for a queue either)
    equal(out[1], out[4])


@pytest.mark.parametrize("narea, nage, seed_E", [(33, 1, 40), (40, 3, 500), (50, 5, 6)])
def test_small_models_with_slots_in_the_queue_s_place(narea, nage, seed_E):
    """Observations of unknown value add slots and nothing else; with 4,000 of them (16 KB) from one run
    to the next, runs of either kind are among those whose state fits."""
    arr, tabs = workload(narea, nage, seed_E)
    want, _ = proposals(arr, tabs, False)
    S = int(arr["dims"][6])
    ran = []
    for n in range(30000, 58000, 4000):
        more = dict(arr)
        for k in [k for k in arr if k.startswith("obs_")]:
            more[k] = np.concatenate([np.asarray(arr[k]).reshape(-1), np.repeat(np.asarray(arr[k]).reshape(-1)[:1], n)])
        nobs, ncell = len(arr["obs_value"]), len(arr["obs_cells"])
        more["obs_sett_i"][nobs:], more["obs_sett_f"][nobs:] = 0, S
        more["obs_value_kind"][nobs:] = 1                  # unknown
        more["obs_cell_ptr"] = np.concatenate([arr["obs_cell_ptr"], ncell + 1 + np.arange(n)]).astype(np.int32)
        try:
            got, _ = proposals(more, tabs, False)
        except capi.BeepError as e:
            assert e.status == 1 and ran                   # too large for the fast form
            break
        equal(got, want)
        ran.append(n)
    assert len(ran) >= 3
