"""Window-sum maps are formed by the passes whose kernels read one and that have
lags enough for it, and by no others."""
import numpy as np
import pytest

from multi_quickpiv_b200 import PIV, correlation_planes, setPIVParameters, synth

pytestmark = pytest.mark.gpu


def _scans(ctx, call):
    """Spans of the integral passes and the map that `call` takes."""
    ctx.profile_enable(True)
    try:
        call()
        return ctx.profile_read()["launches_integral"]
    finally:
        ctx.profile_enable(False)


# FFT lengths 32, 64 (strips, one warp per area), 128 and 256 on both sides of their lines (lags a position; small
# images); with SN strips alone read one (steps up to the window, at most 36 lag rows)
CASES_2D = [(512, "nsqecc", 16, 8, 10, False, True), (512, "nsqecc", 16, 8, 24, False, False),
            (1536, "nsqecc", 32, 16, 24, False, True), (1536, "nsqecc", 32, 16, 64, False, False),
            (512, "nsqecc", 32, 16, 40, False, True), (640, "nsqecc", 32, 10, 32, False, False),
            (1536, "nsqecc", 64, 32, 32, False, True), (1536, "nsqecc", 64, 32, 128, False, False),
            (512, "nsqecc", 64, 32, 64, False, True),
            (1800, "nsqecc", 100, 60, 60, False, True), (1800, "nsqecc", 100, 60, 250, False, False),
            (512, "nsqecc", 32, 16, 8, True, True), (512, "nsqecc", 32, 16, 33, True, False),
            (512, "nsqecc", 12, 19, 12, True, False), (512, "nsqecc", 64, 32, 32, True, False),
            (1536, "zncc", 24, 16, 32, False, True), (1536, "zncc", 24, 16, 64, False, False),
            (512, "zncc", 24, 16, 24, True, False), (512, "fft", 32, 16, 8, False, False)]


@pytest.mark.parametrize("n,alg,IS,SM,st,sn,formed", CASES_2D)
def test_2d(n, alg, IS, SM, st, sn, formed, gpu):
    import torch
    i1, i2, _ = synth.pair_2d_shift(shape=(n, n), shift=(2.6, -3.3), seed_stream=61, dtype=np.float32)
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (i1, i2)]
    p = setPIVParameters(corr_alg=alg, interSize=(IS, IS), searchMargin=(SM, SM), step=(st, st), computeSN=sn)
    assert _scans(gpu, lambda: PIV(*d, p)) == {"fft": 0, "nsqecc": 1, "zncc": 2}[alg] + formed


def test_planes_take_none(gpu):
    i1, i2, _ = synth.pair_2d_shift(shape=(200, 180), shift=(2.6, -3.3), seed_stream=62, dtype=np.float32)
    p = setPIVParameters(corr_alg="nsqecc", interSize=(32, 32), searchMargin=(16, 16), step=(4, 4))
    assert _scans(gpu, lambda: correlation_planes(i1, i2, p, 0, 600)) == 1


@pytest.mark.parametrize("alg,IS,SM,st,sn,formed", [
    ("nsqecc", 16, 8, 8, False, True), ("nsqecc", 16, 8, 40, False, False), ("nsqecc", 16, 8, 8, True, False),
    ("nsqecc", 24, 16, 12, False, True), ("nsqecc", 24, 16, 36, False, False), ("nsqecc", 24, 16, 18, False, False),
    ("zncc", 16, 8, 8, False, True), ("zncc", 16, 8, 40, False, False), ("fft", 16, 8, 8, False, False)])
def test_3d(alg, IS, SM, st, sn, formed, gpu):
    import torch
    i1, i2, _ = synth.pair_3d_shear(shape=(96, 96, 96), seed_stream=63, dtype=np.float32)
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (i1, i2)]
    p = setPIVParameters(corr_alg=alg, interSize=(IS,) * 3, searchMargin=(SM,) * 3, step=(st,) * 3, computeSN=sn)
    assert _scans(gpu, lambda: PIV(*d, p)) == {"fft": 0, "nsqecc": 1, "zncc": 1}[alg] + formed
