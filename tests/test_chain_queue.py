"""Where MBP proposals queue their draws: never at the price of a round more of
an SM's chains; and the counts of a chain do not depend on it."""
import ctypes as C
import itertools
import os
import subprocess

import numpy as np
import pytest

from beep_gb300 import build as bb, capi, model_builder as mb, synth

KB = 1024


@pytest.fixture(scope="module")
def fits(tmp_path_factory):
    tmp = str(tmp_path_factory.mktemp("queue"))
    with open(os.path.join(tmp, "rule.cc"), "w") as f:
        f.write('#include "beep_internal.h"\nextern "C" int fits(size_t s, size_t q, int most, int per_sm)\n'
                '{ return beep::chain_queue_fits(s, q, most, per_sm); }\n')
    so = os.path.join(tmp, "rule.so")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(bb.nvcc()))), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", bb.CSRC, "-I", cuda,
                    os.path.join(tmp, "rule.cc"), "-o", so], check=True)
    L = C.CDLL(so)
    L.fits.argtypes = [C.c_size_t, C.c_size_t, C.c_int, C.c_int]
    return L.fits


def test_rule(fits):
    def rounds(b, most, per_sm):
        n = min(most, 228 * KB // (b + KB))
        return -(-per_sm // n)

    for s, q, most, n in itertools.product(range(4, 228, 7), (17, 35, 87), (1, 2, 3, 4), (1, 2, 3, 4, 5, 8)):
        want = s + q <= 227 and rounds((s + q) * KB, most, n) <= rounds(s * KB, most, n)
        assert bool(fits(s * KB, q * KB, most, n)) == want, (s, q, most, n)
    assert fits(100 * KB, 35 * KB, 2, 1) and not fits(100 * KB, 35 * KB, 2, 2)
    assert not fits(50 * KB, 17 * KB, 4, 4) and fits(50 * KB, 17 * KB, 4, 3)


@pytest.mark.gpu
@pytest.mark.parametrize("narea, nage", [(100, 1), (120, 2), (51, 5)])
def test_counts_of_few_and_many_chains(narea, nage):
    w = synth.seir_hd_small(seed=20261200 + narea, narea=narea, nage=nage, days=20, steps_per_day=2)
    w.obs_kind = "hosp_pop"
    w.seed_E[:, :] = 60
    m = capi.Model(mb.model_arrays(w))
    tabs = [[capi.Tables(mb.param_tables_batch(w, [r], [4.0], [5.0])[0])] for r in (2.4, 2.7)]
    out = []
    for nc in (16, 152, 304, 608):
        dm = capi.DeviceModel(m)
        ch = capi.MbpChains(dm, nc, form=capi.FORM_FAST)
        so = np.arange(nc, dtype=np.uint32)
        ch.initialise(tabs[0], 9, stream_of=so)
        L = ch.propose(tabs[1], 9, stream_of=so + 1000)
        ch.accept(np.ones(nc, np.uint8))
        out.append(([ch.read_state(k) for k in range(16)], L[:16]))
        ch.close()
        dm.close()
    for st, L in out[1:]:
        for (n0, m0), (n1, m1) in zip(out[0][0], st):
            assert np.array_equal(n0, n1) and np.array_equal(m0, m1)
        np.testing.assert_allclose(L, out[0][1], rtol=1e-6)
