"""Single-pair 3D passes (z-spectra shared per layer, window-sum maps, the
approximate peak walk) against batch plans (spectra per area, the full
similarity of every lag): the same fields bit for bit, at chunk, layer and
window edges."""
import numpy as np
import pytest

from multi_quickpiv_b200 import PIV, _lib, setPIVParameters, synth

pytestmark = pytest.mark.gpu


def _both(i1, i2, sn=False, **kw):
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
        np.testing.assert_allclose(SN.cpu().numpy(), SNb.cpu().numpy(), rtol=1e-11)
    plan.close()
    return VF.cpu().numpy()


# (volume, interSize, margin, step): FFT lengths 32, 64 and 128, clipped on every side, odd sizes, one
# layer and several, windows that do not overlap (spectra not shared)
CASES = [((40, 37, 33), (16,) * 3, (8,) * 3, (5, 7, 6)), ((70, 66, 68), (32,) * 3, (16,) * 3, (16, 16, 20)),
         ((50, 61, 24), (12, 17, 9), (9, 3, 6), (12, 8, 5)), ((96, 70, 65), (24, 30, 20), (12, 17, 22), (24, 20, 20)),
         ((130, 90, 80), (48, 40, 36), (24, 20, 20), (40, 25, 30)), ((64, 64, 64), (32,) * 3, (16,) * 3, (32,) * 3)]


@pytest.mark.parametrize("alg", ["fft", "nsqecc", "zncc"])
@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("sn,dtype", [(False, np.float32), (False, np.float64), (True, np.float32)])
def test_equal_batch_plan(alg, case, sn, dtype, gpu):
    shape, IS, SM, st = case
    i1, i2, _ = synth.pair_3d_shear(shape=shape, seed_stream=43, dtype=dtype)
    VF = _both(i1, i2, sn, corr_alg=alg, interSize=IS, searchMargin=SM, step=st)
    assert np.isfinite(VF).all()


@pytest.mark.parametrize("alg", ["fft", "nsqecc", "zncc"])
def test_ties_skips_chunks(alg, gpu):
    """Constant and empty volumes, a periodic pattern, skipped areas, a predictor
    pass, and chunks of one area to several layers."""
    g = np.random.default_rng(5)
    kw = dict(corr_alg=alg, interSize=(16,) * 3, searchMargin=(8,) * 3, step=(8,) * 3)
    flat = np.full((40, 44, 36), 3.0, dtype=np.float32)
    _both(flat, flat, **kw)
    _both(flat * 0, flat * 0, **kw)
    tile = np.tile(g.uniform(0, 9, (4, 4, 4)).astype(np.float32), (10, 11, 9))
    _both(tile, tile, **kw)
    i1, i2, _ = synth.pair_3d_shear(shape=(40, 44, 36), seed_stream=44)
    i1 = i1.copy()
    i1[:20, :20, :20] = -1.0
    VF = _both(i1, i2, threshold=0.0, **kw)
    assert np.all(VF[:, 0, 0, 0] == 0)
    _both(i1, i2, multipass=2, refine=True, **kw)
    ctx = _lib.default_context(0)
    whole = PIV(i1, i2, setPIVParameters(**kw))[0]
    try:
        for chunk in (1, 7, 19):
            assert ctx.lib.mqp_set_tuning(ctx.handle, _lib.MQP_TUNE_CHUNK3D, chunk) == 0
            assert np.array_equal(PIV(i1, i2, setPIVParameters(**kw))[0], whole)
    finally:
        ctx.lib.mqp_set_tuning(ctx.handle, _lib.MQP_TUNE_CHUNK3D, 0)
