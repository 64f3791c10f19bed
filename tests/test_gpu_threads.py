"""Calls of several contexts at once, as the serving runtime's worker and its
callers make them: kernels whose shared memory varies with the parameters
launch from every thread, whatever the others launch."""
import ctypes as C
import threading

import numpy as np
import pytest

from multi_quickpiv_b200 import _lib, setPIVParameters
from multi_quickpiv_b200.piv import _colmajor_torch

pytestmark = pytest.mark.gpu


# (interSize, margin, step) per thread: strips of four areas, whose rows grow with the step; the one-warp
# kernel (a step above the window) at the smallest and largest lag box; the 128-point kernel likewise
@pytest.mark.parametrize("configs", [
    [(32, 16, 8), (32, 16, 31)],
    [(31, 1, 32), (20, 17, 21)],
    [(64, 32, 32), (40, 44, 24)],
])
def test_contexts_in_threads(configs, gpu):
    import torch
    lib, n = _lib.load(), 768
    g = np.random.default_rng(1)
    img = _colmajor_torch(torch.from_numpy(g.uniform(0, 9, (n, n)).astype(np.float32)).cuda())
    torch.cuda.synchronize()
    failed = []

    def call(k, ctx, VF, stream):
        IS, SM, st = configs[k]
        p = setPIVParameters(corr_alg="nsqecc", interSize=(IS, IS), searchMargin=(SM, SM), step=(st, st))
        p.ndims = 2
        cp = p.to_c()
        return lib.mqp_piv_device(ctx.handle, C.c_void_p(img.data_ptr()), C.c_void_p(img.data_ptr()), None, None,
                                  _lib.MQP_F32, 2, (C.c_int64 * 3)(n, n, 1), C.byref(cp), C.c_void_p(VF.data_ptr()),
                                  None, C.c_void_p(stream.cuda_stream))

    def field(k):
        nv = (n - configs[k][0]) // configs[k][2] + 1
        return torch.full((nv, nv, 2), float("nan"), dtype=torch.float64, device="cuda")

    alone = [field(k) for k in range(len(configs))]
    for k, VF in enumerate(alone):
        _lib.check(call(k, gpu, VF, torch.cuda.default_stream()), gpu.handle)
    torch.cuda.synchronize()
    assert all(torch.isfinite(VF).all() for VF in alone)

    def calls(k):
        ctx, VF, stream = _lib.Context(0), field(k), torch.cuda.Stream()
        stream.wait_stream(torch.cuda.default_stream())
        start.wait()
        for _ in range(2000):
            if call(k, ctx, VF, stream) != _lib.MQP_OK:
                failed.append((configs[k], lib.mqp_last_error(ctx.handle).decode()))
                break
        stream.synchronize()
        if not torch.equal(VF, alone[k]):
            failed.append((configs[k], "another field than the call's alone"))
        ctx.close()

    start = threading.Barrier(len(configs))
    threads = [threading.Thread(target=calls, args=(k,)) for k in range(len(configs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
