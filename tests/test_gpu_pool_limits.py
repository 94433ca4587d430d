"""What a model and a server keep of finished batches' buffers: at most 256 MiB
after batches that are each larger or larger together, and none that a waiting
request needs within the server's budget."""
import time

import numpy as np
import pytest

from beep_gb300 import capi, model_builder as mb, synth

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.fixture(scope="module")
def small():
    w = synth.seir_hd_small(seed=20261201, narea=12, nage=3, days=40, steps_per_day=2)
    m = capi.Model(mb.model_arrays(w))
    return m, [capi.Tables(mb.param_tables_batch(w, [2.5], [4.0], [5.0])[0])]


def used(torch):
    free, total = torch.cuda.mem_get_info()
    return total - free


def trajectories(m, tabs, P):
    """69 kB of counts per particle, on the device and pinned."""
    return capi.Batch(m, tabs, P, 1, want_transnum=True, form=capi.FORM_FAST)


def test_a_model_keeps_at_most_its_share(small):
    torch = pytest.importorskip("torch")
    m, tabs = small
    dm = capi.DeviceModel(m)
    dm.simulate(trajectories(m, tabs, 4))
    base = used(torch)
    for P in (5000, 2000, 2500, 3000, 6000, 1000):          # 345, 138, 173, 207, 415, 69 MB
        dm.simulate(trajectories(m, tabs, P))
        assert used(torch) - base <= 256 * MB + 32 * MB, P   # (the driver's own granularity beside them)
    dm.close()
    assert used(torch) - base <= 32 * MB


def test_spare_buffers_make_room_for_the_oldest_request(small):
    torch = pytest.importorskip("torch")
    m, tabs = small
    w = synth.seir_hd_small(seed=20261202, narea=120, nage=6, days=300, steps_per_day=4)
    slow = capi.Model(mb.model_arrays(w))
    slow_tab = [capi.Tables(mb.param_tables_batch(w, [2.5], [4.0], [5.0])[0])]
    base = used(torch)
    srv = capi.Server(640 * MB, 3)
    want = trajectories(m, tabs, 5500)
    dm = capi.DeviceModel(m)
    dm.simulate(want)
    dm.close()
    for _ in range(2):
        slow_run = srv.submit(slow, capi.Batch(slow, slow_tab, 4, 2), capi.REQ_LIKELIHOOD)
        first = trajectories(m, tabs, 4500)                 # 311 MB, spare while the slow one runs
        k = srv.submit(m, first, capi.REQ_SCENARIO)
        srv.wait(k, 60.0)
        second = trajectories(m, tabs, 5500)                # 380 MB: more than the 311 spare leave
        k2 = srv.submit(m, second, capi.REQ_SCENARIO)
        srv.wait(k2, 60.0)
        srv.wait(slow_run, 60.0)
        assert np.array_equal(second.transnum, want.transnum)
        assert np.array_equal(first.transnum, want.transnum[:4500])
        st = [srv.stats(x) for x in (k, k2, slow_run)]
        assert sum(s["device_bytes"] for s in st[1:]) <= 640 * MB
        for x in (k, k2, slow_run):
            srv.release(x)
    time.sleep(0.2)
    assert used(torch) - base <= 256 * MB + 64 * MB          # idle
    srv.close()
    assert used(torch) - base <= 64 * MB
