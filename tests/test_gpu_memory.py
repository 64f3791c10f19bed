"""A context's window-sum map, which its passes can do without, gives way to a
buffer that finds no memory."""
import ctypes as C

import numpy as np
import pytest

from multi_quickpiv_b200 import _lib, setPIVParameters, synth
from multi_quickpiv_b200.piv import _colmajor_torch

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_map_gives_way(gpu):
    import torch
    shape, IS, SM, st = (200, 200, 160), 16, 8, 8
    i1, i2, _ = synth.pair_3d_shear(shape=shape, seed_stream=71, dtype=np.float32)
    d = [_colmajor_torch(torch.from_numpy(np.ascontiguousarray(x)).cuda()) for x in (i1, i2)]
    nv = [(s - IS) // st + 1 for s in shape]
    VF, SN = (torch.zeros(nv[::-1] + k, dtype=torch.float64, device="cuda") for k in ([3], []))

    def call(ctx, budget, sn=False):
        p = setPIVParameters(corr_alg="nsqecc", interSize=(IS,) * 3, searchMargin=(SM,) * 3, step=(st,) * 3, computeSN=sn)
        p.ndims = 3
        cp = p.to_c()
        ctx.set_chunk3d(0, budget)
        VF.fill_(float("nan"))
        _lib.check(ctx.lib.mqp_piv_device(ctx.handle, C.c_void_p(d[0].data_ptr()), C.c_void_p(d[1].data_ptr()), None, None,
                                          _lib.MQP_F32, 3, (C.c_int64 * 3)(*shape), C.byref(cp), C.c_void_p(VF.data_ptr()),
                                          C.c_void_p(SN.data_ptr()) if sn else None, None), ctx.handle)
        torch.cuda.synchronize()
        return VF.cpu().numpy()

    other = _lib.Context(0)  # every kernel loaded, with and without a map
    whole = call(other, 96 * MB)
    assert np.array_equal(call(other, 96 * MB, sn=True), whole)
    other.close()
    ctx = _lib.Context(0)
    assert np.array_equal(call(ctx, 16 * MB), whole)  # 65 MB of integral volume, 52 of map, up to 16 of chunks
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - 40 * MB, dtype=torch.uint8, device="cuda")
    try:
        # 96 MB of chunks find 40 + 16 free, and 52 with the map's
        assert np.array_equal(call(ctx, 96 * MB), whole)
    finally:
        del hog
        torch.cuda.empty_cache()
        ctx.close()
