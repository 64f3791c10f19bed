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


def test_top_two(emu):
    """The two largest values and the largest's lag, however the lags are split;
    of equal maxima the merge keeps a lag of one and counts both."""
    g = np.random.default_rng(5)
    for n, lanes in ((1, 1), (7, 32), (441, 32), (1089, 128), (4225, 128)):
        for v in (g.uniform(-1, 1, n), np.round(g.uniform(0, 3, n)), -np.ones(n)):
            v = np.ascontiguousarray(v, dtype=np.float32)
            b1, b2, idx = C.c_float(), C.c_float(), C.c_int()
            emu.mqp_walk_top(n, lanes, _p(v), C.byref(b1), C.byref(b2), C.byref(idx))
            top = np.sort(np.maximum(np.append(v, [0, 0]), 0))[::-1]  # values above 0 alone count
            assert (b1.value, b2.value) == (top[0], top[1])
            assert (idx.value == -1 and top[0] == 0) or v[idx.value] == top[0]


def test_mapped_windows(emu):
    """Over every area of small axes, moved by every predictor that keeps it
    inside: up to the last mapped lag the map's entry is the lag's window, and in
    range; past it the window ends short of the map's."""
    for size, IS, SM, st in ((9, 4, 3, 2), (16, 5, 8, 3), (12, 12, 4, 1), (40, 8, 8, 5), (33, 16, 1, 7)):
        for v in range((size - IS) // st + 1):
            for d in range(-v * st, size - IS - v * st + 1):
                box, win, mp = np.zeros(4, np.int32), np.zeros((2 * SM + 1, 2), np.int32), np.zeros((2 * SM + 1, 3), np.int32)
                emu.mqp_walk_axis(v, st, IS, SM, size, d, _p(box), _p(win), _p(mp))
                lo, hi, last, ld = box
                assert 0 <= lo <= hi <= 2 * SM
                for s in range(lo, hi + 1):
                    if s <= last:
                        assert 0 <= mp[s, 0] < ld and tuple(win[s]) == tuple(mp[s, 1:]), (size, IS, SM, v, d, s)
                    else:
                        assert win[s, 1] < mp[s, 2]


def test_unmapped_lags(emu):
    """Every lag of the box past the mapped rows or columns, once."""
    for lo1, hi1, lo2, hi2 in ((0, 4, 0, 6), (2, 5, 3, 3), (1, 1, 0, 8)):
        for e1 in range(lo1 - 2, hi1 + 2):
            for e2 in range(lo2 - 2, hi2 + 2):
                hit = np.zeros((9, 6), np.int32)  # [s2, s1]
                emu.mqp_walk_unmapped(lo1, hi1, lo2, hi2, min(e1, hi1), min(e2, hi2), 6, _p(hit))
                s2, s1 = np.indices(hit.shape)
                box = (s1 >= lo1) & (s1 <= hi1) & (s2 >= lo2) & (s2 <= hi2)
                assert np.array_equal(hit, (box & ((s1 > e1) | (s2 > e2))).astype(np.int32)), (lo1, hi1, lo2, hi2, e1, e2)


@pytest.mark.parametrize("P1,P2", [(129, 129), (3, 200), (191, 5), (193, 7)])
def test_huge_tiles(emu, P1, P2):
    """Columns and lag rows of the 256-point kernel through its shared-memory
    tiles (lag rows up to 191) equal those read straight from the scratch slot,
    and the correlation that the spectra stand for."""
    g = np.random.default_rng(P1)
    x, y = g.normal(size=(256, 256)), np.zeros((256, 256))  # search window [x1, x2], interrogation window
    y[:128, :128] = g.normal(size=(128, 128))
    X, Y = np.fft.fft(x, axis=1), np.fft.fft(y, axis=1)  # along dim 2: rows of [x1][k2]

    def packed(S, rows):  # [k2][x1], k2 = 0 and 128 (real) share column 0
        out = S[:rows, :128].T.copy()
        out[0] = S[:rows, 0].real + 1j * S[:rows, 128].real
        return np.ascontiguousarray(np.stack([out.real, out.imag], -1), dtype=np.float32)

    G, F = packed(X, 256), packed(Y, 128)
    lag = [np.zeros((P2, P1), np.float32) for _ in range(2)]
    for tiled in (0, 1):
        emu.mqp_huge_columns(_p(G), _p(F), P1, P2, tiled, _p(lag[tiled]))
    assert np.array_equal(lag[0], lag[1])
    c = np.fft.irfft2(np.conj(np.fft.rfft2(y)) * np.fft.rfft2(x), (256, 256))[:P1, :P2].T
    scale = np.sum(c * lag[0]) / np.sum(c * c)
    # FP32 transforms of length 256 in both directions: relative error of the plane below 1e-6 of its norm
    assert np.linalg.norm(lag[0] / scale - c) < 1e-6 * np.linalg.norm(c)


@pytest.mark.parametrize("M", [32, 64])
def test_packed_product(emu, M):
    """conj(F) G of two real rows' spectra carried in one column as A + iB."""
    g = np.random.default_rng(M)
    a, b, u, v = (np.fft.fft(g.normal(size=2 * M)) for _ in range(4))
    two = lambda z: np.ascontiguousarray(np.stack([z.real, z.imag], -1), dtype=np.float32)
    G, F, out = two(a + 1j * b), two(u + 1j * v), np.zeros((2 * M, 2), np.float32)
    emu.mqp_packed_column(M, _p(G), _p(F), _p(out))
    ref = np.conj(u) * a + 1j * np.conj(v) * b
    assert np.max(np.abs(out[:, 0] + 1j * out[:, 1] - ref)) < 16 * EPS32 * np.max(np.abs(ref)) * 4
