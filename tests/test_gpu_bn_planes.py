"""fp32 batch-norm kernels by planes (16-byte loads where planes allow them, several blocks per plane, gradient with an addend,
statistics whose fp32 sums cancel) against double precision."""
import ctypes as C

import numpy as np
import pytest

from arraydiff_cuda_b200 import abi
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _put(a, gap, lift):
    """A view of planes whose rows are `gap` floats apart, behind a base `lift` floats off 16 bytes."""
    import torch
    N, Cc, Hh, W = a.shape
    n = N * Cc * Hh * (W + gap)
    flat = torch.full((n + 8,), 3.0, device="cuda")
    t = flat[lift:lift + n].view(N, Cc, Hh, W + gap)
    t[..., :W] = H.dev(a)
    return flat, t, abi.Tensor4(t.data_ptr(), abi.AD_F32, N, Cc, Hh, W, *t.stride())


def _beside(flat, t, lift, W):
    """Everything of the buffer but the view's elements is untouched."""
    import torch
    rest = flat.clone()
    rest[lift:lift + t.numel()].view(t.shape)[..., :W] = 3.0
    return torch.all(rest == 3.0).item()


def _reference(x, dy, gamma, beta, relu, mean, invstd):
    """Both passes in 64 bits with the statistics that they are given, and the size of what the ReLU sees."""
    x, dy = x.astype(np.float64), dy.astype(np.float64)
    sh = (1, -1, 1, 1)
    n = x.shape[0] * x.shape[2] * x.shape[3]
    xhat = (x - mean.reshape(sh)) * invstd.reshape(sh)
    pre = gamma.reshape(sh) * xhat + beta.reshape(sh)
    g = np.where(pre <= 0, 0.0, dy) if relu else dy
    db, dg = g.sum((0, 2, 3)), (g * xhat).sum((0, 2, 3))
    dx = gamma.reshape(sh) * invstd.reshape(sh) * (g - db.reshape(sh) / n - xhat * dg.reshape(sh) / n)
    return np.maximum(pre, 0) if relu else pre, dx, dg, db, np.abs(pre)


# planes of whole vectors: one block, a partial last block of 2048, images that share a split; others: the same with blocks of 1024;
# rows apart, bases off 16 bytes; planes of a few pixels, many of them
PLANES = [
    ((1, 5, 2, 2), 0, 0), ((3, 4, 6, 6), 0, 0), ((2, 3, 28, 76), 0, 0), ((7, 2, 50, 82), 0, 0), ((5, 700, 8, 9), 0, 0),
    ((3, 4, 5, 7), 0, 0), ((2, 3, 31, 67), 0, 0), ((9, 2, 45, 47), 0, 0),
    ((2, 3, 20, 60), 4, 0), ((2, 3, 40, 31), 1, 0), ((3, 4, 6, 6), 0, 1), ((2, 3, 28, 76), 0, 2),
    ((33, 40, 1, 1), 0, 0), ((16, 130, 7, 7), 0, 0), ((8, 520, 2, 2), 0, 0), ((4, 6, 1, 3), 0, 0),
    ((3, 130, 1, 5), 0, 0), ((2, 65, 16, 16), 0, 0), ((2, 65, 4, 65), 0, 0), ((5, 67, 16, 17), 0, 1), ((5, 67, 3, 43), 2, 0),   # several planes per block, a last block of fewer
]


@pytest.mark.parametrize("relu", [0, 1])
@pytest.mark.parametrize("shape,gap,lift", PLANES)
def test_bn_planes(shape, gap, lift, relu):
    import torch
    N, Cc, Hh, W = shape
    x, dy, old = H.normal(1, shape) + H.uniform(2, (1, Cc, 1, 1)), H.normal(3, shape), H.normal(4, shape)
    gamma, beta = H.uniform(5, (Cc,), 0.5, 1.5), H.normal(6, (Cc,), 0.3)
    # a pixel within a rounding of the ReLU's edge may fall on either side of it: no gradient there
    x64, sh = x.astype(np.float64), (1, Cc, 1, 1)
    m64, v64 = x64.mean((0, 2, 3)), x64.var((0, 2, 3))
    dy[np.abs(gamma.reshape(sh) * (x64 - m64.reshape(sh)) / np.sqrt(v64 + 1e-5).reshape(sh) + beta.reshape(sh)) < 1e-4] = 0
    (fx, tx, vx), (fdy, tdy, vdy), (fo, to, vo) = (_put(a, gap, lift) for a in (x, dy, old))
    (fy, ty, vy), (fd, td, vd) = _put(np.zeros(shape, np.float32), gap, lift), _put(old, gap, lift)
    g_, b_ = H.dev(gamma), H.dev(beta)
    mean, invstd, var, dg, db = (torch.ones(Cc, device="cuda") for _ in range(5))
    L = abi.lib()
    scratch = torch.full((L.ad_bn_scratch_bytes(Cc),), 255, dtype=torch.uint8, device="cuda")
    sp, sb = H.ptr(scratch), scratch.numel()
    abi.check(L.ad_bn_fwd_train(C.byref(vx), C.byref(vy), H.ptr(g_), H.ptr(b_), H.ptr(mean), H.ptr(invstd), H.ptr(var), 1e-5, relu, sp, sb, H.stream()))
    H.sync()
    # sums whose rounding reaches 1e-6 of the spread (of the variance) are replaced by double ones; then one rounding
    assert np.all(np.abs(H.host(mean) - m64) < 1.1e-6 * np.sqrt(v64) + 1e-7 * np.abs(m64))
    assert np.all(np.abs(H.host(var) - v64) < 1.2e-6 * v64)
    m, i = H.host(mean).astype(np.float64), H.host(invstd).astype(np.float64)
    y_w, dx_w, dg_w, db_w, mag = _reference(x, dy, gamma, beta, relu, m, i)
    size_y = mag + 1 + (np.abs(gamma * i) * np.abs(m)).max()
    assert np.all(np.abs(H.host(ty)[..., :W] - y_w) <= 1e-6 * size_y)
    for addend, base, acc in ((None, 0.0, 0), (vo, old, 0), (vd, None, 1)):
        before = H.host(td)[..., :W].astype(np.float64)
        dg.fill_(1.0), db.fill_(1.0)
        abi.check(L.ad_bn_bwd_add(C.byref(vx), C.byref(vdy), C.byref(addend) if addend is not None else None, C.byref(vd), H.ptr(g_), H.ptr(b_), H.ptr(mean),
                                  H.ptr(invstd), H.ptr(dg), H.ptr(db), relu, acc, sp, sb, H.stream()))
        H.sync()
        want = dx_w + (before if base is None else base)
        size = np.abs(gamma * i).max() * (np.abs(dy).max() + 1) + np.abs(want).max()
        assert np.max(np.abs(H.host(td)[..., :W] - want)) < 2e-6 * size
        tol = 2e-6 * np.abs(dy).sum((0, 2, 3)) + 1e-6
        assert np.all(np.abs(H.host(db) - acc - db_w) < tol) and np.all(np.abs(H.host(dg) - acc - dg_w) < 5 * tol)
    assert all(_beside(f, t, lift, W) for f, t in ((fx, tx), (fdy, tdy), (fo, to), (fy, ty), (fd, td)))
    # fixed statistics through the same planes
    abi.check(L.ad_bn_fwd_inference(C.byref(vx), C.byref(vy), H.ptr(g_), H.ptr(b_), H.ptr(mean), H.ptr(var), H.ptr(invstd), 1e-5, relu, H.stream()))
    H.sync()
    assert np.all(np.abs(H.host(ty)[..., :W] - y_w) <= 2e-6 * size_y)


@pytest.mark.parametrize("shape,gap", [((2, 6, 40, 52), 0), ((4, 3, 33, 45), 0), ((1, 600, 12, 12), 0), ((2, 3, 24, 30), 2)])
def test_bn_planes_mean_far_above_the_spread(shape, gap):
    """Mean 100, spread 0.1: E[x^2] - E[x]^2 of fp32 sums keeps no digit of the variance; that of the double ones does."""
    import torch
    N, Cc, Hh, W = shape
    x, dy = H.normal(1, shape, 0.1) + 100.0 + H.uniform(2, (1, Cc, 1, 1)), H.normal(3, shape)
    x = x.astype(np.float32)
    gamma, beta = H.uniform(5, (Cc,), 0.5, 1.5), H.normal(6, (Cc,), 0.3)
    (_, tx, vx), (_, tdy, vdy) = _put(x, gap, 0), _put(dy, gap, 0)
    (_, ty, vy), (_, td, vd) = (_put(np.zeros(shape, np.float32), gap, 0) for _ in range(2))
    g_, b_ = H.dev(gamma), H.dev(beta)
    mean, invstd, var, dg, db = (torch.zeros(Cc, device="cuda") for _ in range(5))     # the sums are added to
    L = abi.lib()
    scratch = torch.full((L.ad_bn_scratch_bytes(Cc),), 255, dtype=torch.uint8, device="cuda")
    sp, sb = H.ptr(scratch), scratch.numel()
    abi.check(L.ad_bn_fwd_train(C.byref(vx), C.byref(vy), H.ptr(g_), H.ptr(b_), H.ptr(mean), H.ptr(invstd), H.ptr(var), 1e-5, 0, sp, sb, H.stream()))
    abi.check(L.ad_bn_bwd(C.byref(vx), C.byref(vdy), C.byref(vd), H.ptr(g_), H.ptr(b_), H.ptr(mean), H.ptr(invstd), H.ptr(dg), H.ptr(db), 0, 0, sp, sb, H.stream()))
    H.sync()
    x64 = x.astype(np.float64)
    m64, v64 = x64.mean((0, 2, 3)), x64.var((0, 2, 3))
    assert np.all(np.abs(H.host(mean) - m64) < 1e-7 * 102)          # the mean's own rounding: 2^-24 of 100
    # the splits' sums are pairs of floats of 48 bits, 2^-48 of 1e4 is 4e-9 of the variance; then one rounding
    assert np.all(np.abs(H.host(var) - v64) < 1e-6 * v64)
    m, i = H.host(mean).astype(np.float64), H.host(invstd).astype(np.float64)
    y_w, dx_w, dg_w, db_w, _ = _reference(x, dy, gamma, beta, 0, m, i)
    # x - mean is exact, what follows rounds at 2^-24 of values of a few spreads
    assert np.max(np.abs(H.host(ty)[..., :W] - y_w)) < 1e-5 and np.max(np.abs(H.host(td)[..., :W] - dx_w)) < 1e-5 * np.abs(dx_w).max()
    scale = np.abs(dy).sum((0, 2, 3))
    assert np.all(np.abs(H.host(db) - db_w) < 1e-5 * scale) and np.all(np.abs(H.host(dg) - dg_w) < 5e-5 * scale)
