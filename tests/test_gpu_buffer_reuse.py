"""Buffers handed from one batch to the next (a model's pool, a server's pool):
results do not depend on what a buffer held before, from one thread or
several, the memory is given back, and a finished request can be released at
once."""
import threading

import numpy as np
import pytest

from beep_gb300 import capi, model_builder as mb, synth

pytestmark = pytest.mark.gpu


def small(narea=12, nage=3, days=40):
    w = synth.seir_hd_small(seed=20260301, narea=narea, nage=nage, days=days, steps_per_day=2)
    rng = np.random.default_rng(1)
    m = capi.Model(mb.model_arrays(w))
    return m, [capi.Tables(t) for t in mb.param_tables_batch(w, *synth.abc_smc_priors(rng, 4))]


def batch(m, tabs, P, seed, form, **kw):
    return capi.Batch(m, tabs, P, seed, group_of=np.arange(P) % 4, want_pop=True, form=form, **kw)


@pytest.mark.parametrize("form", [capi.FORM_PLAIN_FP64, capi.FORM_FAST])
def test_batches_of_changing_sizes_reuse_buffers(form):
    m, tabs = small()
    sizes = [300, 7, 299, 1, 64, 300]
    want = []
    for k, P in enumerate(sizes):
        dm = capi.DeviceModel(m)                      # a pool of its own, nothing to reuse
        want.append(dm.simulate(batch(m, tabs, P, k, form, want_transnum=k % 2 == 0)))
        dm.close()
    dm = capi.DeviceModel(m)

    def run():
        for k, P in enumerate(sizes):
            g = dm.simulate(batch(m, tabs, P, k, form, want_transnum=k % 2 == 0))
            assert np.array_equal(g.L, want[k].L) and np.array_equal(g.pop, want[k].pop)
            if k % 2 == 0:
                assert np.array_equal(g.transnum, want[k].transnum)
    run()
    errors = []

    def guarded():
        try:
            run()
        except BaseException as e:                    # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=guarded) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    dm.close()


def test_memory_is_given_back():
    import torch
    m, tabs = small()
    dm = capi.DeviceModel(m)
    dm.simulate(batch(m, tabs, 8, 1, capi.FORM_FAST))
    dm.close()
    free0 = torch.cuda.mem_get_info()[0]
    dm = capi.DeviceModel(m)
    for P in (20000, 30000):                          # beyond what a model keeps: 30000 x 80 steps of counts
        dm.simulate(capi.Batch(m, tabs, P // 20, 1, want_transnum=True, form=capi.FORM_FAST))
    assert free0 - torch.cuda.mem_get_info()[0] <= 600 << 20
    dm.close()
    assert free0 - torch.cuda.mem_get_info()[0] <= 64 << 20


def test_finished_requests_are_released_at_once():
    m, tabs = small(10, 2, 30)
    dm = capi.DeviceModel(m)
    want = [dm.simulate(batch(m, tabs, 5 + k, k, capi.FORM_FAST)) for k in range(8)]
    dm.close()
    srv = capi.Server(1 << 30, 4)
    for k in range(160):
        b = batch(m, tabs, 5 + k % 8, k % 8, capi.FORM_FAST)
        t = srv.submit(m, b, capi.REQ_LIKELIHOOD)
        srv.wait(t, 60.0)
        srv.release(t)
        assert np.array_equal(b.L, want[k % 8].L) and np.array_equal(b.pop, want[k % 8].pop)
    srv.close()
