"""CPU check of the approximate peak walk's parts (mqp_finish.cuh), compiled for
the host: tests/native/mqp_emu_walk.cu."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

NATIVE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")
CSRC = os.path.join(os.path.dirname(os.path.dirname(NATIVE)), "multi_quickpiv_b200", "csrc")
EPS32 = 2.0 ** -24


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("walk") / "libmqp_walk.so")
    subprocess.run(["nvcc", "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC,-fvisibility=hidden",
                    "-shared", "-I", CSRC, os.path.join(NATIVE, "mqp_emu_walk.cu"), "-o", out], check=True)
    return C.CDLL(out)


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def _nsqecc(emu, S2, c, F2):
    S2, c = np.ascontiguousarray(S2, dtype=np.float64), np.ascontiguousarray(c, dtype=np.float32)
    walk, full = np.zeros(len(S2)), np.zeros(len(S2))
    is_open = emu.mqp_walk_nsqecc(len(S2), _p(S2), _p(c), C.c_double(F2), _p(walk), _p(full))
    return is_open, walk, full


@pytest.mark.parametrize("F2", [1e-29, 3.7, 1e9, 9e29])
def test_nsqecc_approximation(emu, F2):
    """Lags whose denominator is at least a quarter of F2 + S2 are within the
    stated bound of the full value; one below it opens the area, whichever
    sign it has."""
    g = np.random.default_rng(3)
    S2 = F2 * 10 ** g.uniform(-9, 7, 4000)
    c = np.float32(np.sqrt(F2 * S2) * g.uniform(-1, 1, 4000))  # Cauchy
    is_open, walk, full = _nsqecc(emu, S2, c, F2)
    assert not is_open
    # 12 roundings to FP32 in the denominator, the reciprocal, the product; 2 in the full value
    assert np.max(np.abs(walk / full - 1)) < 16 * EPS32
    for part, expect in ((0.26, 0), (0.24, 1), (1e-4, 1), (-1e-7, 1), (-0.3, 1)):
        # the transforms' error takes the denominator to `part` of F2 + S2
        s2 = F2 * g.uniform(0.5, 2)
        bad = np.float32((F2 + s2 + np.sqrt(F2 * s2) - part * (F2 + s2)) / 2)
        at = g.integers(0, 4000)
        S2b, cb = S2.copy(), c.copy()
        S2b[at], cb[at] = s2, bad
        assert _nsqecc(emu, S2b, cb, F2)[0] == expect


@pytest.mark.parametrize("F2", [1e-29, 3.7, 9e29])
def test_masked_approximation(emu, F2):
    """Masked lags within the bound keep the full value; a cancelled denominator
    opens the area also where the approximate root leaves it negative."""
    g = np.random.default_rng(4)
    S2 = F2 * 10 ** g.uniform(-6, 6, 4000) * np.where(g.uniform(size=4000) < 0.1, -1, 1)  # the transforms' error has no sign
    d = np.sqrt(np.abs(S2) * F2)
    share = g.uniform(0.3, 3, 4000) * np.where(g.uniform(size=4000) < 0.3, -1, 1)  # denominator / d
    c1 = (F2 + S2 + d - share * d) / 2
    emu.mqp_walk_masked.restype = C.c_float

    def run(c1):
        walk, full = np.zeros(4000), np.zeros(4000)
        return emu.mqp_walk_masked(4000, _p(S2), _p(c1), C.c_double(F2), _p(walk), _p(full)), walk, full

    most, walk, full = run(c1)
    assert most <= 4
    assert np.max(np.abs(walk / full - 1)) < 4 * EPS32  # the same denominator; reciprocal and product against a quotient
    for part in (0.1, 1e-3, 1e-6, -1e-6, -1e-3, -0.1):
        cb, at = c1.copy(), g.integers(0, 4000)
        cb[at] = (F2 + S2[at] + d[at] - part * d[at]) / 2
        assert run(cb)[0] > 4
