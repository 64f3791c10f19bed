"""The single-pair 2D passes against the work-queue kernel of batch plans (one
warp per interrogation area, integral-image lookups at every lag): the same
fields bit for bit, at the sizes where strips, window-sum maps and the
approximate peak walk have edges."""
import numpy as np
import pytest

from multi_quickpiv_b200 import PIV, setPIVParameters, synth

pytestmark = pytest.mark.gpu


def _both(i1, i2, sn, **kw):
    import torch
    from multi_quickpiv_b200.batch import BatchPlan
    p = setPIVParameters(computeSN=sn, **kw)
    d1, d2 = torch.from_numpy(np.ascontiguousarray(i1)).cuda(), torch.from_numpy(np.ascontiguousarray(i2)).cuda()
    VF, SN = PIV(d1, d2, p)
    plan = BatchPlan([(d1, d2, p)], options={"use_graph": 0})
    plan.run()
    torch.cuda.synchronize()
    VFb, SNb = plan.results()[0]
    assert np.array_equal(VF.cpu().numpy(), VFb.cpu().numpy(), equal_nan=True)
    if sn:
        # the FP64 sum of the plane runs over the lanes in another order
        np.testing.assert_allclose(SN.cpu().numpy(), SNb.cpu().numpy(), rtol=1e-11)
    plan.close()
    return VF.cpu().numpy()


# (image, interSize, margin, step): strips of one to five areas, margins from one lag row to the
# direct-sum rows (33..36) and past them, windows clipped on every side, anisotropic sizes
SHAPES = [((64, 64), (32, 32), (16, 16), (8, 8)), ((203, 177), (32, 32), (16, 16), (8, 8)),
          ((260, 99), (32, 32), (10, 10), (32, 32)), ((131, 140), (24, 31), (18, 9), (5, 31)),
          ((300, 64), (20, 32), (17, 16), (7, 3)), ((90, 210), (33, 12), (1, 20), (9, 12)),
          ((150, 150), (12, 30), (19, 2), (12, 30)), ((512, 520), (32, 32), (16, 16), (7, 8)),
          ((97, 101), (16, 16), (8, 8), (3, 5))]


@pytest.mark.parametrize("alg", ["fft", "nsqecc", "zncc"])
@pytest.mark.parametrize("case", SHAPES)
@pytest.mark.parametrize("sn", [False, True])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_equal_work_queue_kernel(alg, case, sn, dtype, gpu):
    shape, IS, SM, st = case
    i1, i2, _ = synth.pair_2d_shift(shape=shape, shift=(2.6, -3.3), seed_stream=41, dtype=dtype)
    VF = _both(i1, i2, sn, corr_alg=alg, interSize=IS, searchMargin=SM, step=st)
    assert np.isfinite(VF).all()


@pytest.mark.parametrize("alg", ["fft", "nsqecc", "zncc"])
def test_ties_skips_and_scales(alg, gpu):
    """Constant images (every lag ties), skipped areas, a periodic pattern
    (several equal maxima) and images whose sums leave the FP32 range."""
    g = np.random.default_rng(3)
    flat = np.full((96, 80), 7.0, dtype=np.float32)
    kw = dict(corr_alg=alg, interSize=(32, 32), searchMargin=(16, 16), step=(8, 8))
    _both(flat, flat, False, **kw)
    noise = g.uniform(1, 2, (96, 80)).astype(np.float32)
    noise[:40, :40] = -1.0
    VF = _both(noise, noise, False, threshold=0.0, **kw)
    assert np.all(VF[:, 0, 0] == 0)
    tile = np.tile(g.uniform(0, 9, (8, 8)).astype(np.float32), (12, 10))
    _both(tile, tile, False, **kw)
    for s in (1e-18, 1e17):
        _both(noise * np.float32(s), noise * np.float32(s), False, **kw)


@pytest.mark.parametrize("IS,SM,st", [(16, 8, 8), (32, 16, 13), (24, 11, 12), (64, 32, 32), (48, 20, 21)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_masked_walk_equals_full_search(IS, SM, st, dtype, gpu):
    """Masked NSQECC without SN (the approximate walk) against the same pass
    with SN (every lag in full), with areas the mask covers fully, partly, by a
    few pixels and not at all."""
    import torch
    i1, i2, _ = synth.pair_2d_shift(shape=(203, 177), shift=(2.6, -3.3), seed_stream=45, dtype=dtype)
    g = np.random.default_rng(9)
    mask = np.zeros(i1.shape, dtype=dtype)
    mask[30:140, 20:120] = 1
    mask[::37, ::29] = 1  # lone pixels
    mask[60:80, 60:80] = g.uniform(0, 1, (20, 20))
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (i1, i2, mask)]
    kw = dict(interSize=(IS, IS), searchMargin=(SM, SM), step=(st, st))
    walk = PIV(*d, setPIVParameters(**kw))[0].cpu().numpy()
    full = PIV(*d, setPIVParameters(computeSN=True, **kw))[0].cpu().numpy()
    assert np.array_equal(walk, full, equal_nan=True)
