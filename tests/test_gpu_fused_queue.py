"""Fused chain launches over sets that queue their draws, sets that have no room
to (the matrix of 166 areas in shared memory) and both together: each set's
counts are those of its own launch."""
import numpy as np
import pytest

from beep_gb300 import capi, model_builder as mb, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [((166, 3),), ((20, 2),), ((166, 3), (20, 2)), ((33, 6), (170, 1), (166, 3))])
def test_fused_as_separate(sizes):
    sets = []
    for narea, nage in sizes:
        w = synth.seir_hd_small(seed=20261300 + narea, narea=narea, nage=nage, days=15, steps_per_day=2)
        w.obs_kind = "hosp_pop"
        w.seed_E[:, :] = 60
        m = capi.Model(mb.model_arrays(w))
        t = [capi.Tables(mb.param_tables_batch(w, [r], [4.0], [5.0])[0]) for r in (2.4, 2.7)]
        sets.append((m, t))
    nc = 7
    so = np.arange(nc, dtype=np.uint32)
    out = []
    for fused in (False, True):
        dms = [capi.DeviceModel(m) for m, _ in sets]
        chs = [capi.MbpChains(dm, nc, form=capi.FORM_FAST) for dm in dms]
        for ch, (_, t) in zip(chs, sets):
            ch.initialise([t[0]], 9, stream_of=so)
        if fused:
            L = capi.MbpChains.propose_fused(chs, [dict(tables=[t[1]], seed=5, stream_of=so + 90) for _, t in sets])
        else:
            L = [ch.propose([t[1]], 5, stream_of=so + 90) for ch, (_, t) in zip(chs, sets)]
        for ch in chs:
            ch.accept(np.ones(nc, np.uint8))
        out.append(([[ch.read_state(k) for k in range(nc)] for ch in chs], L))
        for ch, dm in zip(chs, dms):
            ch.close()
            dm.close()
    for (sa, La), (sb, Lb) in [((a, la), (b, lb)) for a, la, b, lb in zip(out[0][0], out[0][1], out[1][0], out[1][1])]:
        for (na, ma), (nb, mb_) in zip(sa, sb):
            assert na.sum() > 0 and np.array_equal(na, nb)
            assert np.array_equal(ma, mb_)
        np.testing.assert_allclose(La, Lb, rtol=1e-6)
