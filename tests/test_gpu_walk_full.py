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
