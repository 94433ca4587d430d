"""The FP32-decided samplers of the plain form (rng_filter.cuh) against the FP64
samplers they stand for, trial by trial on chosen words: at every place where a
decision turns -- between two counts, and between accepting and rejecting one --
and at distances from it below and above the filter's bounds.  The counts
include 0 and n (the ends of the binomial's density) and those around 10 (the
Poisson's change from log k! to its series).  On the CPU with the approximate
operations off by their documented errors to either side; on the GPU with the
operations themselves."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from beep_gb300 import build as bb

HERE = os.path.dirname(os.path.abspath(__file__))
TRIAL = np.dtype([("par", "f8"), ("n", "i4"), ("x", "u4"), ("y", "u4"), ("fp64", "i4")], align=True)


def headers(tmp):
    """Copies of the samplers' headers whose Philox block is the key (then, for a second trial, words beyond
    the density's peak with a V near 0): the words of a draw as arguments."""
    src = open(os.path.join(bb.CSRC, "rng_fp64.cuh")).read()
    name = "__device__ __forceinline__ U4 philox10(U4 c, uint32_t k0, uint32_t k1)"
    assert src.count(name) == 1
    own = ("__device__ __forceinline__ U4 philox10(U4 c, uint32_t k0, uint32_t k1)\n"
           "{ return c.w & 0xffffu ? U4{k0 >> 31 ? 0x60000000u : 0xA0000000u, 0u, 0u, 0u} : U4{k0, k1, 0u, 0u}; }\n")
    src = src.replace(name, own + name.replace("philox10", "philox10_keyed"))
    with open(os.path.join(tmp, "rng_fp64.cuh"), "w") as f:
        f.write(src)
    shutil.copy(os.path.join(bb.CSRC, "rng_filter.cuh"), tmp)
    shutil.copy(os.path.join(HERE, "filtered_draws.cu"), tmp)


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    tmp = str(tmp_path_factory.mktemp("filtered"))
    headers(tmp)
    so = os.path.join(tmp, "host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-w", "-x", "c++",
                    "filtered_draws.cu", "-o", so], cwd=tmp, check=True)
    L = C.CDLL(so)
    L.boundary_trials.restype = C.c_int64
    L.boundary_trials.argtypes = [C.c_double, C.c_int32, C.c_void_p, C.c_int, C.c_void_p, C.c_int64]
    L.filtered_host.argtypes = [C.c_void_p, C.c_int64, C.c_int, C.c_void_p]
    L.filtered_host.restype = None
    L.fp64_host.argtypes = [C.c_void_p, C.c_int64]
    L.fp64_host.restype = None
    return L, tmp


def boundaries(L, par, n, counts):
    buf = np.zeros(200000, TRIAL)
    want = np.array(sorted(set(int(k) for k in counts)), np.int32)
    m = L.boundary_trials(par, n, want.ctypes.data, len(want), buf.ctypes.data, len(buf))
    assert 0 < m < len(buf)
    return buf[:m]


def poisson_cases():
    rng = np.random.default_rng(1)
    for mean in [1e-3, 0.3, 1.0, 4.0, 9.99, 10.0, 10.7, 12.0, 15.5, 23.0, 60.0, 333.3, 4e3, 1e5, 3.3e6, 8e8,
                 *np.exp(rng.uniform(np.log(0.01), np.log(1e7), 12))]:
        sd = np.sqrt(mean)
        near = np.floor(mean + sd * rng.uniform(-5, 5, 8))
        yield mean, -1, [k for k in [0, 1, 2, 5, 8, 9, 10, 11, 12, 15, *near] if 0 <= k <= mean + 6 * sd + 2]


def binomial_cases():
    rng = np.random.default_rng(2)
    for n in (20, 21, 25, 40, 100, 101, 1000, 30000, 10**6, 5 * 10**8):
        for nq in (0.4, 6.0, 9.99, 10.0, 10.05, 10.08, 10.11, 11.0, 12.5, 14.0, 0.37 * n, 0.5 * n):
            if nq > 0.5 * n:
                continue
            for p in (nq / n, 1.0 - nq / n):
                q = min(p, 1.0 - p)
                sd = np.sqrt(n * q * (1 - q))
                near = np.floor(n * q + sd * rng.uniform(-5, 5, 6))
                yield p, n, [k for k in [0, 1, 2, 3, n - 2, n - 1, n, *near] if 0 <= k <= n]


def philox(c, k0, k1):
    c = list(c)
    for _ in range(10):
        a, b = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
        c = [(b >> 32) ^ c[1] ^ k0, b & 0xffffffff, (a >> 32) ^ c[3] ^ k1, a & 0xffffffff]
        k0, k1 = (k0 + 0x9E3779B9) & 0xffffffff, (k1 + 0xBB67AE85) & 0xffffffff
    return c


def all_trials(L):
    parts = [boundaries(L, *c) for c in poisson_cases()] + [boundaries(L, *c) for c in binomial_cases()]
    return np.concatenate(parts)


def report(t, got):
    bad = np.nonzero(t["fp64"] != got)[0]
    return len(bad), [(tuple(t[k].tolist()), int(got[k])) for k in bad[:5]]


@pytest.mark.parametrize("off", range(5))
def test_trials_at_the_bounds(host, off):
    L, _ = host
    t = all_trials(L)
    got = np.empty(len(t), np.int32)
    L.filtered_host(t.ctypes.data, len(t), off, got.ctypes.data)
    assert np.array_equal(t["fp64"], got), report(t, got)


def test_a_binomial_draw_of_zero(host):
    """100 x 0.1008 under key (1234, 0), column 19598974, transition 3, step 111, stream 7: a first
    trial of 0, accepted by 1e-4 of the density's logarithm."""
    L, _ = host
    w = philox((19598974, 111, 7, (4 << 24) | (3 << 16)), 1234, 0)
    t = np.array([(0.1008, 100, w[0], w[1], 0)], TRIAL)
    got = np.empty(1, np.int32)
    L.filtered_host(t.ctypes.data, 1, 4, got.ctypes.data)
    assert got[0] == 0


@pytest.mark.parametrize("mean", (0.999e9, 1.001e9, 2.147e9, 2.2e9, 5e9, 1e12, float("inf")))
def test_means_around_and_beyond_32_bits(host, mean):
    """The draws' words at random: the FP64 sampler's counts, whatever it makes of a mean beyond them."""
    L, _ = host
    rng = np.random.default_rng(5)
    t = np.zeros(2000, TRIAL)
    t["par"], t["n"] = mean, -1
    t["x"], t["y"] = rng.integers(0, 1 << 32, (2, len(t)), dtype=np.uint32)
    L.fp64_host(t.ctypes.data, len(t))
    got = np.empty(len(t), np.int32)
    for off in range(5):
        L.filtered_host(t.ctypes.data, len(t), off, got.ctypes.data)
        assert np.array_equal(t["fp64"], got), report(t, got)


@pytest.mark.gpu
def test_trials_at_the_bounds_gpu(host):
    L, tmp = host
    so = os.path.join(tmp, "gpu.so")
    subprocess.run([bb.nvcc()] + bb.ARCH + ["-O3", "-std=c++17", "--fmad=false", "-Xcompiler", "-fPIC", "-shared",
                    "filtered_draws.cu", "-o", so], cwd=tmp, check=True)
    G = C.CDLL(so)
    G.filtered_gpu.argtypes = [C.c_void_p, C.c_longlong, C.c_void_p]
    t = all_trials(L)
    got = np.empty(len(t), np.int32)
    assert G.filtered_gpu(t.ctypes.data, len(t), got.ctypes.data) == 0
    assert np.array_equal(t["fp64"], got), report(t, got)
