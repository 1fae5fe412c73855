"""Vector batch-norm kernels (any multiple of 8 channels, second stage of the statistics, gradient with an addend) against
the oracle."""
import ctypes as C

import numpy as np
import pytest

from arraydiff_cuda_b200 import abi
from oracle import orc
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [
    (1, 8, 1, 1),          # one pixel: a single partial row
    (2, 24, 5, 7),         # channel groups that do not divide the block
    (1, 64, 90, 61),       # several blocks
    (2, 344, 33, 31), (1, 2048, 9, 11), (3, 2040, 17, 13),
    (2, 64, 210, 211),     # the full grid
])
@pytest.mark.parametrize("pad", [0, 1])
def test_bn_vector_forms(shape, pad):
    import torch
    N, Cc, Hh, W = shape
    x, dy, old = (orc.round_bf16(H.normal(i, shape)) for i in (1, 2, 3))
    gamma, beta = H.uniform(4, (Cc,), 0.5, 1.5), H.normal(5, (Cc,), 0.3)
    y_w, mean_w, invstd_w, var_w = orc.bn_fwd_train(x, gamma, beta, relu=True, omp=True)
    L = abi.lib()

    def put(a):
        t = torch.full((N, Hh + 2 * pad, W + 2 * pad, Cc), 3.0, dtype=torch.bfloat16, device="cuda")
        t[:, pad:pad + Hh, pad:pad + W] = H.dev_bf16(orc.nchw_to_nhwc(a))
        return t, H.view_nhwc(t, (pad, Hh, W))

    def get(t):
        return orc.nhwc_to_nchw(H.host(t)[:, pad:pad + Hh, pad:pad + W])

    (tx, vx), (tdy, vdy), (told, vold) = put(x), put(dy), put(old)
    ty, vy = put(np.zeros(shape, np.float32))
    tdx, vdx = put(old)
    g_, b_ = H.dev(gamma), H.dev(beta)
    mean, invstd, var, dg, db = (torch.ones(Cc, device="cuda") for _ in range(5))
    scratch = torch.full((L.ad_bn_scratch_bytes(Cc),), 255, dtype=torch.uint8, device="cuda")
    sp, sb = H.ptr(scratch), scratch.numel()
    for _ in range(2):                     # again on the same scratch
        abi.check(L.ad_bn_fwd_train(C.byref(vx), C.byref(vy), H.ptr(g_), H.ptr(b_), H.ptr(mean), H.ptr(invstd), H.ptr(var), 1e-5, 1, sp, sb, H.stream()))
    H.sync()
    n = N * Hh * W
    assert H.max_rel(H.host(mean), mean_w) < 1e-5 or np.max(np.abs(H.host(mean) - mean_w)) < 1e-6
    if n > 1:
        assert H.max_rel(H.host(invstd), invstd_w) < 1e-5 and H.max_rel(H.host(var), var_w) < 1e-5
    assert np.max(np.abs(get(ty) - y_w)) < 2e-2 * max(1.0, np.max(np.abs(y_w)))
    assert np.all(H.host(ty)[:, :pad] == 3.0)
    if n == 1:
        return
    m, i = H.host(mean), H.host(invstd)
    dx_w, dg_w, db_w = orc.bn_bwd(x, dy, gamma, beta, m, i, relu=True, omp=True)
    args = [H.ptr(g_), H.ptr(b_), H.ptr(mean), H.ptr(invstd), H.ptr(dg), H.ptr(db), 1]
    scale = max(1.0, np.max(np.abs(dx_w)))
    for addend, want, acc in ((None, dx_w, 0), (vold, dx_w + old, 0), (vdx, None, 1)):
        before = get(tdx)
        dg.fill_(1.0), db.fill_(1.0)
        abi.check(L.ad_bn_bwd_add(C.byref(vx), C.byref(vdy), C.byref(addend) if addend is not None else None, C.byref(vdx), *args, acc, sp, sb, H.stream()))
        H.sync()
        want = before + dx_w if want is None else want
        assert np.max(np.abs(get(tdx) - want)) < 2e-2 * max(scale, np.max(np.abs(want)))
        assert H.max_rel(H.host(dg) - acc, dg_w) < 1e-4 and H.max_rel(H.host(db) - acc, db_w) < 1e-4
    assert np.array_equal(H.host(told), H.host(put(old)[0]))      # an addend is only read
    assert L.ad_bn_bwd_add(C.byref(vx), C.byref(vdy), C.byref(H.view_nhwc(told[:, :, :, :Cc // 2])), C.byref(vdx), *args, 0, sp, sb, H.stream()) == abi.AD_ERR_BAD_ARG
