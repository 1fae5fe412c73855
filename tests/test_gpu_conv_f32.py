"""Tiled fp32 convolution kernels against the oracle, at the edges of their tiles, splits and tap classes."""
import ctypes as C

import numpy as np
import pytest

from arraydiff_cuda_b200 import abi
from oracle import orc
from tests import helpers as H
from tests.test_gpu_conv import conv_args

pytestmark = pytest.mark.gpu

CASES = [
    # N, C, H, W, K, k, stride, dil, pad
    (1, 1, 1, 1, 1, 1, 1, 1, 0),         # one output
    (1, 3, 23, 29, 33, 3, 1, 1, 1),      # a row past the 32-row tile
    (2, 65, 9, 13, 65, 3, 1, 2, 2),      # a row past the 64-row tile, reduction split over a cluster
    (3, 16, 31, 33, 129, 1, 1, 1, 0),    # 1x1, a row past the 128-row tile
    (1, 8, 97, 131, 24, 3, 2, 1, 1),     # strided: four classes of gradient pixels, unequal tap counts
    (2, 6, 15, 14, 7, 2, 3, 1, 0),       # stride above the filter: classes without any tap
    (1, 5, 21, 22, 9, 3, 2, 2, 1),       # strided and dilated: taps of one class only
    (1, 3, 40, 44, 64, 7, 1, 1, 3),      # 49 taps
    (4, 40, 120, 118, 48, 3, 1, 1, 0),   # no cluster split forward; filter gradient in slices of the scratch
    (2, 24, 130, 129, 20, 3, 1, 1, 1),   # 32-row tiles
    (1, 17, 60, 61, 16, 5, 1, 1, 2),     # 16-row tiles
    (2, 9, 70, 50, 8, 3, 1, 1, 1),       # 8-row tiles: a row per CTA of a cluster of 8
    (1, 96, 100, 101, 128, 3, 1, 1, 1),  # two 64-row tiles
    (1, 128, 7, 9, 130, 3, 1, 1, 1),     # clusters of 16 forward and in the data gradient (test_clusters_of_16)
    (1, 120, 8, 9, 16, 3, 1, 1, 1),      # forward: a row of the 16-row tile per CTA
]


@pytest.mark.parametrize("tiles", [None, "1", "0"])   # by size, the tiled kernels, a thread per output
@pytest.mark.parametrize("case", CASES)
def test_conv_f32_tiles(case, tiles, monkeypatch):
    import torch
    if tiles:
        monkeypatch.setenv("ARRAYDIFF_B200_F32_TILES", tiles)
    N, Cc, Hh, W, K, k, s, d, pd = case
    x, w, b = H.uniform(1, (N, Cc, Hh, W)), H.normal(2, (K, Cc, k, k), float(np.sqrt(2.0 / (k * k * Cc)))), H.normal(3, (K,))
    y_w = orc.conv2d_fprop(x, w, b, (s, s), (d, d), (pd, pd), omp=True)
    dy = H.uniform(4, y_w.shape)
    dx_w = orc.conv2d_dgrad(dy, w, x.shape, (s, s), (d, d), (pd, pd), omp=True)
    db_w = np.zeros(K, np.float32)
    dw_w = orc.conv2d_wgrad(x, dy, w.shape, (s, s), (d, d), (pd, pd), db=db_w, omp=True)
    L = abi.lib()
    a = conv_args(abi.AD_F32, abi.AD_NCHW, x.shape, K, k, s, d, pd)
    dx_, dw_, db_, ddy = H.dev(x), H.dev(w), H.dev(b), H.dev(dy)
    P, Q = y_w.shape[2:]
    # y and dy as views into wider rows, as a strip inside a padded buffer is
    y, gy = torch.full((N, K, P + 1, Q + 3), 7.0, device="cuda"), torch.full((N, K, P + 1, Q + 3), float("nan"), device="cuda")
    gy[:, :, :P, :Q] = ddy
    a.x, a.w, a.bias, a.y, a.relu = dx_.data_ptr(), dw_.data_ptr(), db_.data_ptr(), y.data_ptr(), 1
    a.y_pitch, a.y_plane = Q + 3, (P + 1) * (Q + 3)
    abi.check(L.ad_conv2d_fprop(C.byref(a), H.stream()))
    gdx, gdw, gdb = torch.ones(x.shape, device="cuda"), torch.full(w.shape, 9.0, device="cuda"), torch.full((K,), 9.0, device="cuda")
    a.y, a.dx, a.dw, a.db, a.accumulate = gy.data_ptr(), gdx.data_ptr(), gdw.data_ptr(), gdb.data_ptr(), 1
    abi.check(L.ad_conv2d_dgrad(C.byref(a), H.stream()))
    a.accumulate = 0
    scratch = torch.full((max(16, L.ad_conv2d_scratch_bytes(C.byref(a), 2)),), 255, dtype=torch.uint8, device="cuda")
    a.scratch, a.scratch_bytes = scratch.data_ptr(), scratch.numel()
    abi.check(L.ad_conv2d_wgrad(C.byref(a), H.stream()))
    H.sync()
    got = H.host(y)
    assert H.max_rel(got[:, :, :P, :Q], np.maximum(y_w, 0)) < 1e-5
    assert np.all(got[:, :, P:, :] == 7.0) and np.all(got[:, :, :, Q:] == 7.0)
    assert H.max_rel(H.host(gdx) - 1, dx_w) < 1e-5
    assert H.max_rel(H.host(gdw), dw_w) < 2e-5
    assert H.max_rel(H.host(gdb), db_w) < 2e-5


@pytest.mark.parametrize("case", [(2, 3, 40, 44, 64, 7, 2, 1, 3), (3, 1, 19, 23, 17, 3, 1, 2, 0), (1, 8, 30, 21, 33, 5, 3, 1, 1), (2, 3, 17, 18, 20, 2, 3, 1, 0),
                                  (5, 8, 129, 131, 16, 7, 1, 1, 3)])   # pieces of 2, 2 and 1 image
@pytest.mark.parametrize("accumulate", [0, 1])
def test_data_gradient_into_few_channels(case, accumulate, monkeypatch):
    """The two-step form that a caller's scratch allows."""
    import torch
    monkeypatch.setenv("ARRAYDIFF_B200_F32_TILES", "1")
    N, Cc, Hh, W, K, k, s, d, pd = case
    w = H.normal(2, (K, Cc, k, k), float(np.sqrt(2.0 / (k * k * Cc))))
    P, Q = ((n + 2 * pd - d * (k - 1) - 1) // s + 1 for n in (Hh, W))
    dy = H.uniform(4, (N, K, P, Q))
    want = orc.conv2d_dgrad(dy, w, (N, Cc, Hh, W), (s, s), (d, d), (pd, pd), omp=True)
    L = abi.lib()
    a = conv_args(abi.AD_F32, abi.AD_NCHW, want.shape, K, k, s, d, pd)
    need = L.ad_conv2d_scratch_bytes(C.byref(a), 1)
    z = P * Q * Cc * k * k * 4
    assert need == min(N, (64 << 20) // z) * z
    scratch, dx = torch.full((need,), 255, dtype=torch.uint8, device="cuda"), torch.ones(want.shape, device="cuda")
    gy = torch.full((N, K, P + 1, Q + 3), float("nan"), device="cuda")
    gy[:, :, :P, :Q] = H.dev(dy)
    dw_ = H.dev(w)
    a.y_pitch, a.y_plane = Q + 3, (P + 1) * (Q + 3)
    a.y, a.w, a.dx, a.scratch, a.scratch_bytes, a.accumulate = gy.data_ptr(), dw_.data_ptr(), dx.data_ptr(), scratch.data_ptr(), need, accumulate
    abi.check(L.ad_conv2d_dgrad(C.byref(a), H.stream()))
    H.sync()
    assert np.max(np.abs(H.host(dx) - accumulate - want)) < 1e-5 * np.max(np.abs(want)) + accumulate * 2e-6


def test_data_gradient_of_more_than_2_32_elements():
    """A large stride: 90 images of 3 x 4000 x 4000 behind maps of 64 x 64, by pieces whose elements 32 bits count."""
    import torch
    N, Cc, Hh, K, k, s, P = 90, 3, 4000, 16, 2, 63, 64
    assert N * Cc * Hh * Hh > 1 << 32 and (Hh - k) // s + 1 == P
    L = abi.lib()
    a = conv_args(abi.AD_F32, abi.AD_NCHW, (N, Cc, Hh, Hh), K, k, s, 1, 0)
    g = torch.Generator(device="cuda").manual_seed(5)
    dy, w = torch.rand((N, K, P, P), generator=g, device="cuda"), torch.rand((K, Cc, k, k), generator=g, device="cuda")
    dx = torch.full((N, Cc, Hh, Hh), float("nan"), device="cuda")
    scratch = torch.full((L.ad_conv2d_scratch_bytes(C.byref(a), 1),), 255, dtype=torch.uint8, device="cuda")
    assert scratch.numel() == 44 * P * P * Cc * k * k * 4       # 44 images have fewer than 2^31 elements, 45 more
    a.y, a.w, a.dx, a.scratch, a.scratch_bytes = dy.data_ptr(), w.data_ptr(), dx.data_ptr(), scratch.data_ptr(), scratch.numel()
    abi.check(L.ad_conv2d_dgrad(C.byref(a), H.stream()))
    for n in range(N):
        want = torch.einsum("kpq,kcij->cpiqj", dy[n].double(), w.double())
        full = torch.zeros((Cc, P * s, P * s), device="cuda")    # the last rows and columns are fewer than a stride
        full[:, :Hh, :Hh] = dx[n]
        got = full.unflatten(1, (P, s))[:, :, :k].unflatten(3, (P, s))[..., :k]
        assert (got - want).abs().max() < 1e-5 * want.max() and torch.count_nonzero(dx[n]) == got.numel()   # zeros elsewhere


K1_CASES = [
    # N, C, H, W (of x), K, stride of 1x1 layers: both directions
    (1, 17, 1, 1, 17, 1),          # one pixel, the smallest channel counts of the 1x1 kernels
    (1, 32, 2, 2, 33, 1),          # one vector of pixels; a row past the 32-row tile, filters of the gradient one by one
    (3, 31, 5, 13, 64, 1),         # planes of 65 pixels: gathers one by one; a channel short of two stages
    (2, 65, 6, 22, 36, 1),         # vectors that cross rows, images that share a tile; a row past the 64-row tile
    (1, 130, 9, 12, 24, 1),        # 32-row tiles, reduction split over a cluster
    (5, 48, 16, 20, 148, 1),       # running sums that restart, three tiles of rows
    (1, 2100, 8, 8, 20, 1),        # the largest clusters, shares of unequal length
    (2, 33, 15, 16, 40, 2),        # 8 x 8 planes of dy: vectors; rows and columns between and past the last that belong to no pixel
    (3, 20, 16, 20, 65, 3),        # 6 x 7
]


@pytest.mark.parametrize("pitched", [0, 1])
@pytest.mark.parametrize("case", K1_CASES)
def test_conv_f32_1x1(case, pitched, monkeypatch):
    """The 1x1 kernels at the edges of their tiles, vectors and splits; dense planes and padded ones; operands off by four bytes."""
    import torch
    monkeypatch.setenv("ARRAYDIFF_B200_F32_TILES", "1")
    N, Cc, Hh, W, K, s = case
    P, Q = (Hh - 1) // s + 1, (W - 1) // s + 1
    x, w, b = H.uniform(1, (N, Cc, Hh, W)), H.normal(2, (K, Cc, 1, 1), float(np.sqrt(2.0 / Cc))), H.normal(3, (K,))
    dy = H.uniform(4, (N, K, P, Q))
    y_w = np.einsum("nchw,kc->nkhw", x[:, :, ::s, ::s].astype(np.float64), w[:, :, 0, 0].astype(np.float64)) + b[None, :, None, None]
    add = float(pitched)             # the padded form accumulates, into ones
    dx_w, mag_x = np.full(x.shape, add), np.full(x.shape, add)
    dx_w[:, :, ::s, ::s] += np.einsum("nkhw,kc->nchw", dy.astype(np.float64), w[:, :, 0, 0].astype(np.float64))
    mag_x[:, :, ::s, ::s] += np.einsum("nkhw,kc->nchw", np.abs(dy), np.abs(w[:, :, 0, 0]))
    # a sum of n products, |terms| t: running sums of 64 and n / 64 partial sums round at 2^-24 of what they hold
    eps = lambda n: (min(n, 64) + n // 64 + 4) * 2.0 ** -24  # noqa: E731
    L = abi.lib()
    a = conv_args(abi.AD_F32, abi.AD_NCHW, x.shape, K, 1, s, 1, 0)
    flat = torch.empty(x.size + 1, device="cuda")
    xd = flat[pitched:pitched + x.size].view(x.shape).copy_(H.dev(x))          # one off: no longer 16-byte aligned
    wflat = torch.empty(w.size + 1, device="cuda")
    wd = wflat[pitched:pitched + w.size].view(w.shape).copy_(H.dev(w))
    bd = H.dev(b)
    ph, pw = P + pitched, Q + 3 * pitched
    y, gy = torch.full((N, K, ph, pw), 7.0, device="cuda"), torch.full((N, K, ph, pw), float("nan"), device="cuda")
    gy[:, :, :P, :Q] = H.dev(dy)
    dx = torch.ones(x.shape, device="cuda")
    a.x, a.w, a.bias, a.y, a.y_pitch, a.y_plane = xd.data_ptr(), wd.data_ptr(), bd.data_ptr(), y.data_ptr(), pw, ph * pw
    abi.check(L.ad_conv2d_fprop(C.byref(a), H.stream()))
    a.y, a.dx, a.accumulate = gy.data_ptr(), dx.data_ptr(), pitched
    abi.check(L.ad_conv2d_dgrad(C.byref(a), H.stream()))
    mag_y = np.einsum("nchw,kc->nkhw", np.abs(x[:, :, ::s, ::s]), np.abs(w[:, :, 0, 0])) + np.abs(b)[None, :, None, None]
    assert (np.abs(y[:, :, :P, :Q].cpu().numpy() - y_w) <= eps(Cc) * mag_y).all()
    assert (np.abs(dx.cpu().numpy() - dx_w) <= eps(K) * mag_x).all()
    assert (y[:, :, P:] == 7).all() and (y[:, :, :, Q:] == 7).all()


K3_CASES = [
    # N, C, H, W (of x), K, pad, stride, dilation of 3x3 layers
    (1, 16, 3, 3, 17, 0, 1, 1),          # one output pixel; the smallest channel counts of the 3x3 kernels
    (1, 17, 6, 4, 33, 0, 1, 1),          # one block of 4 x 2 pixels; a channel past a pair of stages, a row past the 32-row tile
    (3, 20, 11, 13, 64, 1, 1, 1),        # blocks past both edges, implicit padding, images that share a tile
    (2, 33, 10, 17, 65, 2, 1, 1),        # padding of 2: the gradient's map is smaller than y; a row past the 64-row tile
    (1, 130, 9, 12, 24, 1, 1, 1),        # 32-row tiles, reduction split over a cluster; rows of 12 = 8 + 4 pixels
    (5, 48, 18, 19, 80, 1, 1, 1),        # running sums that restart, 19 = 8 + 8 + 3 pixels
    (1, 300, 23, 25, 40, 0, 1, 1),       # more than 256 channels per CTA of a cluster of one
    (4, 64, 58, 61, 32, 0, 1, 1),  # filter gradient in clusters and slices of the scratch
    (1, 16, 3, 3, 17, 0, 2, 1),    # one output pixel of stride 2
    (2, 33, 18, 18, 96, 0, 2, 1),  # 8 x 8 pixels; a row and a column of x that no tap meets
    (3, 21, 17, 33, 64, 1, 2, 1),  # 9 x 17: blocks past both edges, rows of 8 + 8 + 1 pixels, implicit padding
    (4, 40, 39, 49, 30, 2, 2, 1),  # 32-row tiles of stride 2; padding of 2
    (2, 20, 20, 21, 64, 2, 1, 2),  # 20 x 21 under dilation 2: maps of 10 x 11 and 10 x 10
    (1, 30, 16, 27, 24, 0, 1, 3),  # 10 x 21: 4, 3 and 3 rows
    (2, 18, 24, 32, 70, 4, 1, 4),  # 24 x 32
    # dilations that the rules send to the 3x3 kernels by themselves, in all three passes and in two
    (2, 64, 32, 32, 64, 2, 1, 2), (2, 64, 48, 48, 64, 3, 1, 3), (1, 64, 64, 64, 70, 4, 1, 4),
    (1, 5, 9, 12, 7, 3, 1, 3),     # fewer channels than a tile has rows; 9 x 12 under dilation 3: maps of 3 x 4
    (1, 20, 11, 3, 18, 4, 1, 4),   # rows of 3 under dilation 4: a map and a segment without pixels
]


# "1": as the rules choose (small maps stay with the general tiles), "2": the 3x3 kernels in every pass that they can serve (all but
# the data gradient of a stride)
@pytest.mark.parametrize("tiles", ["1", "2"])
@pytest.mark.parametrize("scratch", [True, False])
@pytest.mark.parametrize("case", K3_CASES)
def test_conv_f32_3x3(case, scratch, tiles, monkeypatch):
    """The 3x3 kernels at the edges of their tiles, blocks, segments and splits, with strides and dilations; infinities stay where they have a weight."""
    import torch
    monkeypatch.setenv("ARRAYDIFF_B200_F32_TILES", tiles)
    N, Cc, Hh, W, K, pd, s, d = case
    x, w, b = H.uniform(1, (N, Cc, Hh, W)), H.normal(2, (K, Cc, 3, 3), float(np.sqrt(2.0 / (9 * Cc)))), H.normal(3, (K,))
    y_w = orc.conv2d_fprop(x, w, b, (s, s), (d, d), (pd, pd), omp=True)
    dy = H.uniform(4, y_w.shape)
    dx_w = orc.conv2d_dgrad(dy, w, x.shape, (s, s), (d, d), (pd, pd), omp=True)
    db_w = np.zeros(K, np.float32)
    dw_w = orc.conv2d_wgrad(x, dy, w.shape, (s, s), (d, d), (pd, pd), db=db_w, omp=True)
    L = abi.lib()
    a = conv_args(abi.AD_F32, abi.AD_NCHW, x.shape, K, 3, s, d, pd)
    P, Q = y_w.shape[2:]
    y, gy = torch.full((N, K, P + 1, Q + 3), 7.0, device="cuda"), torch.full((N, K, P + 1, Q + 3), float("nan"), device="cuda")
    gy[:, :, :P, :Q] = H.dev(dy)
    xd, wd, bd = H.dev(x), H.dev(w), H.dev(b)
    dx, dw, db = torch.ones(x.shape, device="cuda"), torch.ones(w.shape, device="cuda"), torch.ones(K, device="cuda")
    a.x, a.w, a.bias, a.y, a.y_pitch, a.y_plane = xd.data_ptr(), wd.data_ptr(), bd.data_ptr(), y.data_ptr(), Q + 3, (P + 1) * (Q + 3)
    abi.check(L.ad_conv2d_fprop(C.byref(a), H.stream()))
    a.y, a.dx, a.dw, a.db, a.accumulate = gy.data_ptr(), dx.data_ptr(), dw.data_ptr(), db.data_ptr(), 1
    abi.check(L.ad_conv2d_dgrad(C.byref(a), H.stream()))
    if scratch:
        part = torch.full((max(16, L.ad_conv2d_scratch_bytes(C.byref(a), 2)),), 255, dtype=torch.uint8, device="cuda")
        a.scratch, a.scratch_bytes = part.data_ptr(), part.numel()
    abi.check(L.ad_conv2d_wgrad(C.byref(a), H.stream()))
    H.sync()
    got = H.host(y)
    assert H.max_rel(got[:, :, :P, :Q], y_w) < 1e-5
    assert np.all(got[:, :, P:, :] == 7.0) and np.all(got[:, :, :, Q:] == 7.0)
    # 1 + v rounds to 2^-24 of its size
    assert np.max(np.abs(H.host(dx) - 1 - dx_w)) < 1e-5 * np.max(np.abs(dx_w)) + 1e-6
    assert np.max(np.abs(H.host(dw) - 1 - dw_w)) < 2e-5 * np.max(np.abs(dw_w)) + 1e-6
    assert np.max(np.abs(H.host(db) - 1 - db_w)) < 2e-5 * np.max(np.abs(db_w)) + 1e-6
    # an infinite pixel of x reaches the outputs and filter entries that it has a product in, and no others
    n, c, iy, ix = N - 1, Cc - 1, Hh - 1, W - 1
    xd[n, c, iy, ix] = float("inf")
    a.y, a.accumulate = y.data_ptr(), 0
    abi.check(L.ad_conv2d_fprop(C.byref(a), H.stream()))
    a.y = gy.data_ptr()
    abi.check(L.ad_conv2d_wgrad(C.byref(a), H.stream()))
    H.sync()
    hit = np.zeros((N, P, Q), bool)
    taps = np.zeros((Cc, 3, 3), bool)
    for i in range(3):
        for j in range(3):
            oy, ox = iy + pd - i * d, ix + pd - j * d
            if 0 <= oy < P * s and 0 <= ox < Q * s and oy % s == 0 and ox % s == 0:
                hit[n, oy // s, ox // s] = taps[c, i, j] = True
    assert np.array_equal(~np.isfinite(H.host(y)[:, :, :P, :Q]).all(1), hit)
    assert np.array_equal(~np.isfinite(H.host(dw)).all(0), taps)
