"""Passes without SN, which search the peak among FP32 approximations, against
the same passes with SN, which evaluate every lag in full: the same fields bit
for bit."""
import numpy as np
import pytest

from multi_quickpiv_b200 import PIV, setPIVParameters

pytestmark = pytest.mark.gpu


def _walk_equals_full(i1, i2, mask=None, **kw):
    import torch
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (i1, i2) + (() if mask is None else (mask,))]
    walk = PIV(*d, setPIVParameters(**kw))[0].cpu().numpy()
    full = PIV(*d, setPIVParameters(computeSN=True, **kw))[0].cpu().numpy()
    assert np.array_equal(walk, full, equal_nan=True), int((walk != full).sum())
    return walk


def _spots(shape, g, n):
    a, b = np.zeros(shape), np.zeros(shape)
    at, peak = g.integers(0, np.array(shape), (n, len(shape))), g.uniform(0.5, 1, n)
    np.add.at(a, tuple(at.T), peak)
    np.add.at(b, tuple(np.minimum(at + 2, np.array(shape) - 1).T), peak)
    return a, b


# FFT lengths 32, 64 (one warp per area: steps above the window, more than 36 lag rows) and 128, 64 in strips
@pytest.mark.parametrize("IS,SM,st", [((16, 16), (8, 8), (5, 9)), ((32, 32), (16, 16), (40, 40)),
                                      ((12, 30), (19, 2), (12, 30)), ((64, 64), (32, 32), (32, 32)),
                                      ((32, 32), (16, 16), (8, 8))])
@pytest.mark.parametrize("scale", [1e-19, 1e-20, 2e-21])
def test_faint_images(IS, SM, st, scale, gpu):
    """Pixels whose correlation lies at the low end of FP32's range: the
    similarities are those of the transforms' own FP32 values."""
    a, b = _spots((437, 391), np.random.default_rng(7), 3400)
    i1, i2 = (a * scale).astype(np.float32), (b * scale).astype(np.float32)
    VF = _walk_equals_full(i1, i2, corr_alg="nsqecc", interSize=IS, searchMargin=SM, step=st)
    assert np.isfinite(VF).mean() > 0.5


@pytest.mark.parametrize("shape,IS,SM,st,seed", [((2048, 2048), 64, 96, 15, 0), ((2048, 2048), 32, 48, 7, 0),
                                                 ((256, 256, 192), 16, 20, 8, 0), ((256, 256, 192), 16, 20, 8, 1)])
def test_bright_pixels_beside_dark_windows(shape, IS, SM, st, seed, gpu):
    """Pixels 1e9 times brighter than the rest: the transforms' error, which
    grows with the whole search window, cancels NSQECC denominators of the
    windows that hold none of them."""
    g, nd = np.random.default_rng(seed), len(shape)
    a = g.uniform(0.5, 1.5, shape)
    b = a.copy()
    b[tuple(g.integers(0, np.array(shape), (int(np.prod(shape)) // (1500 if nd == 2 else 20000), nd)).T)] = 1e9
    _walk_equals_full(a.astype(np.float32), b.astype(np.float32), corr_alg="nsqecc", interSize=(IS,) * nd,
                      searchMargin=(SM,) * nd, step=(st,) * nd)


# FFT lengths 32, 64 (strips, one warp per area), 128 and 256 in 2D; 32, 64 and 128 in 3D
@pytest.mark.parametrize("shape,IS,SM,st", [((437, 391), 16, 8, 6), ((437, 391), 32, 16, 9), ((437, 391), 24, 12, 25),
                                            ((437, 391), 64, 30, 21), ((437, 391), 100, 60, 50),
                                            ((101, 93, 85), 16, 8, 8), ((101, 93, 85), 32, 16, 15),
                                            ((101, 93, 85), 40, 25, 20)])
@pytest.mark.parametrize("alg", ["nsqecc", "zncc", "mask"])
@pytest.mark.parametrize("kind", ["noise", "period", "flat"])
def test_near_ties(shape, IS, SM, st, alg, kind, gpu):
    """Noise on a bright background, whose similarities lie within a few
    rounding steps of one another, several equal maxima, and every lag equal."""
    nd, g = len(shape), np.random.default_rng(11)
    if alg == "mask" and IS == 100:
        pytest.skip("no masks above 128")
    if kind == "noise":
        i1, i2 = 3000 + 20 * g.uniform(size=shape), 3000 + 20 * g.uniform(size=shape)
    elif kind == "period":
        i1 = np.tile(g.uniform(0, 9, (8,) * nd), [s // 8 + 1 for s in shape])[tuple(slice(0, s) for s in shape)]
        i2 = i1
    else:
        i1 = i2 = np.full(shape, 7.0)
    mask = (g.uniform(size=shape) < 0.7).astype(np.float32) if alg == "mask" else None
    _walk_equals_full(i1.astype(np.float32), i2.astype(np.float32), mask, corr_alg="nsqecc" if alg == "mask" else alg,
                      interSize=(IS,) * nd, searchMargin=(SM,) * nd, step=(st,) * nd)
