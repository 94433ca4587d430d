"""Models whose shared memory is nearly full, in batches small enough for draws
per (transition, column): the layout is taken only where its array of changes
fits too, so that such models run as they do with it switched off (the same
counts' populations and log-likelihoods), or are refused in both."""
import numpy as np
import pytest

from beep_gb300 import capi, model_builder as mb, synth

pytestmark = pytest.mark.gpu


def run_both(arr, t, P):
    m = capi.Model(arr)
    dm = capi.DeviceModel(m)
    out = []
    for opt in (1, 0):                                  # never, automatic
        capi.set_option("fast_parallel_draws", opt)
        try:
            r = dm.simulate(capi.Batch(m, [t], P, 3, want_pop=True, form=capi.FORM_FAST))
            out.append((r.L.copy(), r.pop.copy()))
        except capi.BeepError as e:
            assert e.status == 1, e                     # BEEP_BAD_INPUT: too large for the fast form
            out.append(None)
        finally:
            capi.set_option("fast_parallel_draws", 0)
    dm.close()
    never, auto = out
    assert (never is None) == (auto is None)
    if never is not None:
        assert np.array_equal(never[0], auto[0]) and np.array_equal(never[1], auto[1])
    return never is not None


def with_observations(arr, n, cells):
    """n observations of one cell each over the whole horizon (a slot each)."""
    S = int(arr["dims"][6])
    out = dict(arr)
    for k in [k for k in arr if k.startswith("obs_")]:
        out[k] = np.repeat(np.asarray(arr[k]).reshape(-1)[:1], n)
    out["obs_sett_i"], out["obs_sett_f"] = np.zeros(n, np.int32), np.full(n, S, np.int32)
    out["obs_value"] = np.full(n, 20.0)
    out["obs_sd"] = np.full(n, 30.0)
    out["obs_cell_ptr"] = np.arange(n + 1, dtype=np.int32)
    out["obs_cells"] = np.asarray(cells, np.int32)[np.arange(n) % len(cells)]
    return out


def test_slots_up_to_the_limit():
    """40 areas, 6 transitions: observation slots from where the matrix, the populations and the
    changes fit to where nothing does, in steps smaller than the changes and their wider reduction."""
    w = synth.seir_hd_small(seed=20260701, narea=40, nage=1, days=4, steps_per_day=1)
    arr = mb.model_arrays(w)
    T = int(arr["dims"][5])
    t = capi.Tables(mb.param_tables_batch(w, [2.5], [4.0], [5.0])[0])
    cells = np.arange(40) * T + 1
    ran = [run_both(with_observations(arr, n, cells), t, 5) for n in range(51200, 58400, 400)]
    assert ran[0] and not ran[-1]


@pytest.mark.parametrize("narea", (218, 220, 222, 224, 226, 230))
def test_few_transitions_many_areas(narea):
    """A model of 2 transitions and 3 compartments whose matrix nearly fills the shared memory."""
    w = synth.seir_hd_small(seed=20260702, narea=narea, nage=1, days=6, steps_per_day=2)
    full = mb.model_arrays(w)
    arr = dict(full)
    dims = np.asarray(full["dims"]).copy()
    dims[4], dims[5] = 3, 2
    arr["dims"] = dims
    arr["trans_from"], arr["trans_to"] = np.array([0, 1], np.int32), np.array([1, 2], np.int32)
    pop = np.zeros((narea, 3, 1))
    pop[:, 0], pop[:, 1] = full["pop_init"][:, 0], 40
    arr["pop_init"] = pop
    arr = with_observations(arr, narea, np.arange(narea) * 2)
    raw = mb.param_tables_batch(w, [2.5], [4.0], [5.0])[0]
    t = capi.Tables(dict(raw, transrate=np.array([[0.0], [0.2]]), infectivity=np.array([0.0, 1.0, 0.0])))
    assert run_both(arr, t, 5)
