"""Particle-filter requests beside others: when one finishes, its memory goes to
the server's pool, so the thread that admits and retires does not wait for the
kernels of the requests still running."""
import time

import pytest

from beep_gb300 import capi, model_builder as mb, synth

pytestmark = pytest.mark.gpu


def model(narea, nage, days, steps_per_day):
    w = synth.seir_hd_small(seed=20260801, narea=narea, nage=nage, days=days, steps_per_day=steps_per_day)
    return capi.Model(mb.model_arrays(w)), capi.Tables(mb.param_tables_batch(w, [2.5], [4.0], [5.0])[0])


def test_a_finished_filter_does_not_hold_up_other_requests():
    big, tb = model(300, 8, 300, 4)                        # 1200 FP64 steps on 8 SMs: a few tenths of a second
    m, t = model(10, 3, 20, 2)
    sections = [(0, 20), (20, 40)]
    srv = capi.Server(8 << 30, 4)

    def filter_request():
        k = srv.submit_pf(m, t, 64, 5, 1, 0.5, sections, form=capi.FORM_FAST)
        srv.wait(k, 60.0)
        srv.release(k)

    def small_request():
        b = capi.Batch(m, [t], 16, 3, form=capi.FORM_FAST)
        k = srv.submit(m, b, capi.REQ_LIKELIHOOD)
        srv.wait(k, 60.0)
        srv.release(k)

    def long_request():
        return srv.submit(big, capi.Batch(big, [tb], 8, 2), capi.REQ_LIKELIHOOD)

    filter_request()                                      # kernels loaded, buffers in the pool
    small_request()
    k = long_request()
    srv.wait(k, 120.0)
    st = srv.stats(k)
    assert st["gpu_end_s"] - st["gpu_start_s"] > 0.1
    k = long_request()
    while srv.stats(k)["state"] != 1:                     # (its kernel is launched before the next is admitted)
        time.sleep(0.001)
    filter_request()
    small_request()                                       # admitted after the filter was retired
    assert srv.stats(k)["state"] == 1                     # the long one still runs
    srv.wait(k, 120.0)
    srv.close()


def test_a_filter_is_charged_what_it_holds():
    m, t = model(30, 4, 40, 2)
    N, S = 400, m.ndivision
    sections = [(k, k + 2) for k in range(0, S, 2)]
    srv = capi.Server(8 << 30, 2)
    big = capi.Batch(m, [t], 3000, 1, want_pop=True)       # its buffers go to the pool: larger than the filter's
    k = srv.submit(m, big, capi.REQ_LIKELIHOOD)
    srv.wait(k, 60.0)
    k = srv.submit_pf(m, t, N, 5, 1, 0.5, sections)
    srv.wait(k, 60.0)
    ncol = m.narea * m.ndemocatpos
    per = 4 * (2 * m.ncomp + m.ntrans) * ncol + 8 * 4 * m.nstrain * m.narea * m.nage   # a particle's work in a section
    assert srv.stats(k)["device_bytes"] >= len(sections) * N * per
    srv.close()
