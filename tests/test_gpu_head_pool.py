"""Bilinear row kernels, per-pixel loss forms, global pooling, linear layer, pooling tiles and the bias gradient against
the oracle, at the edges of their blocks and tiles."""
import ctypes as C

import numpy as np
import pytest

from arraydiff_cuda_b200 import abi
from oracle import orc
from tests import helpers as H
from tests.test_gpu_conv import conv_args

pytestmark = pytest.mark.gpu
FMT = {"f32": (abi.AD_F32, abi.AD_NCHW, H.view_nchw), "bf16": (abi.AD_BF16, abi.AD_NHWC, H.view_nhwc)}


def _dev(a, dtype):
    return H.dev(a) if dtype == "f32" else H.dev_bf16(orc.nchw_to_nhwc(a))


def _host(t, dtype):
    a = H.host(t)
    return a if dtype == "f32" else orc.nhwc_to_nchw(a)


def _q(a, dtype):
    return a if dtype == "f32" else orc.round_bf16(a)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("shape,scale", [
    ((1, 1, 1, 1), 2), ((2, 3, 1, 5), 3), ((1, 19, 9, 40), 8), ((2, 150, 3, 37), 4),    # wide classes: several chunks per row
    ((1, 2, 4, 700), 8), ((3, 5, 7, 4), 5), ((1, 64, 5, 33), 1),
])
def test_upsample_rows(dtype, shape, scale):
    import torch
    N, Cc, Hh, W = shape
    x = _q(H.normal(1, shape), dtype)
    dy = _q(H.normal(2, (N, Cc, Hh * scale, W * scale)), dtype)
    y_w, dx_w = orc.upsample_bilinear_fwd(x, scale), orc.upsample_bilinear_bwd(dy, scale)
    _, _, view = FMT[dtype]
    dx_, ddy = _dev(x, dtype), _dev(dy, dtype)
    y, gx = torch.empty_like(ddy), torch.ones_like(dx_)
    vx, vy, vdy, vgx = view(dx_), view(y), view(ddy), view(gx)
    L = abi.lib()
    abi.check(L.ad_upsample_bilinear_fwd(C.byref(vx), C.byref(vy), scale, 0, Hh, 0, H.stream()))
    abi.check(L.ad_upsample_bilinear_bwd(C.byref(vdy), C.byref(vgx), scale, 0, Hh, 0, 1, H.stream()))
    H.sync()
    tol = 1e-5 if dtype == "f32" else 1e-2
    assert H.max_rel(_host(y, dtype), y_w) < tol
    assert H.max_rel(_host(gx, dtype), 1 + dx_w) < tol


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("shape,scale", [((1, 256, 2, 273), 4), ((2, 256, 3, 290), 4), ((1, 1500, 3, 21), 1), ((1, 1500, 2, 31), 1)])
def test_upsample_rows_last_chunk_of_one_column(dtype, shape, scale):
    """Rows cut into chunks (of 17 columns, of 5) whose last has one column, so that the one before ends at the last but one: it has
    all of its row in shared memory and the table of columns right behind (of fewer words than a column has channels)."""
    import torch
    N, Cc, Hh, W = shape
    x = _q(H.normal(1, shape), dtype)
    want = orc.upsample_bilinear_fwd(x, scale)
    t = (H.dev if dtype == "f32" else H.dev_bf16)(orc.nchw_to_nhwc(x))
    y = torch.empty((N, Hh * scale, W * scale, Cc), dtype=t.dtype, device="cuda")
    vx, vy = H.view_nhwc(t), H.view_nhwc(y)
    abi.check(abi.lib().ad_upsample_bilinear_fwd(C.byref(vx), C.byref(vy), scale, 0, Hh, 0, H.stream()))
    H.sync()
    # two blends of two values: a rounding of each, and bf16's own
    assert H.max_rel(orc.nhwc_to_nchw(H.host(y)), want) < (1e-6 if dtype == "f32" else 8e-3)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("layout", [abi.AD_NCHW, abi.AD_NHWC])
@pytest.mark.parametrize("Cc,W,scale", [(19, 40, 8), (3, 300, 4), (1, 1100, 2), (31, 70, 4), (2, 33, 16), (64, 18, 8), (5, 300, 2),
                                        (36, 25, 8), (107, 21, 4)])   # 6 blocks of 4 columns and one of the last, 5 and one
def test_upsample_cells_of_strips(dtype, layout, Cc, W, scale):
    """Rows between two source rows as one block: cells cut by the strips, rows that start on odd elements, odd channel counts, one
    thread group per block (64 channels at scale 8); every element of the strip and none beside it."""
    import torch
    N, Hh = 2, 5
    x = _q(H.normal(1, (N, Cc, Hh, W)), dtype)
    want = orc.upsample_bilinear_fwd(x, scale)
    YW = W * scale
    nchw = layout == abi.AD_NCHW
    tx = H.dev(x).to(torch.float32 if dtype == "f32" else torch.bfloat16)
    tx = tx if nchw else tx.permute(0, 2, 3, 1).contiguous()
    es = abi.AD_F32 if dtype == "f32" else abi.AD_BF16
    for y0, rows, odd in [(0, Hh * scale, 0), (0, scale + 1, 1), (scale // 2 + 1, 2 * scale, 0), ((Hh - 1) * scale + 1, scale - 1, 1)]:
        pitch = YW * (1 if nchw else Cc) + odd
        buf = torch.full((N, Cc if nchw else 1, rows, pitch), 7.0, dtype=tx.dtype, device="cuda")
        if nchw:
            vx = abi.Tensor4(tx.data_ptr(), es, N, Cc, Hh, W, Cc * Hh * W, Hh * W, W, 1)
            vy = abi.Tensor4(buf.data_ptr(), es, N, Cc, rows, YW, Cc * rows * pitch, rows * pitch, pitch, 1)
        else:
            vx = abi.Tensor4(tx.data_ptr(), es, N, Cc, Hh, W, Hh * W * Cc, 1, W * Cc, Cc)
            vy = abi.Tensor4(buf.data_ptr(), es, N, Cc, rows, YW, rows * pitch, 1, pitch, Cc)
        abi.check(abi.lib().ad_upsample_bilinear_fwd(C.byref(vx), C.byref(vy), scale, 0, Hh, y0, H.stream()))
        H.sync()
        got = H.host(buf)
        assert np.all(got[..., pitch - odd:] == 7.0)
        got = got[..., :pitch - odd]
        got = got if nchw else np.transpose(got.reshape(N, rows, YW, Cc), (0, 3, 1, 2))
        # two blends of two values: a rounding of each, and bf16's own
        assert H.max_rel(got, want[:, :, y0:y0 + rows]) < (1e-6 if dtype == "f32" else 8e-3)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("shape,scale", [((1, 3, 6, 40), 8), ((2, 3, 5, 90), 3), ((1, 19, 5, 33), 2), ((1, 1, 4, 700), 5), ((1, 2, 5, 9), 2)])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_upsample_rows_of_infinities(dtype, shape, scale, bad):
    """Logits masked with an infinity, at the right and lower edge and inside, and gradients that overflowed: each reaches the
    elements that it has a weight in and no other (weights of 0 multiply nothing but the next source row and column)."""
    import torch
    N, Cc, Hh, W = shape

    def weights(n):                                  # [output][source], of the half-pixel rule
        o = np.arange(n * scale)
        src = np.maximum((o + 0.5) / scale - 0.5, 0.0)
        i0 = np.minimum(np.floor(src + 1e-9).astype(int), n - 1)
        f = np.where(src - i0 < 1e-9, 0.0, src - i0)
        w = np.zeros((n * scale, n))
        np.add.at(w, (o, i0), 1 - f)
        np.add.at(w, (o, np.minimum(i0 + 1, n - 1)), f)
        touch, zero = w > 0, np.zeros_like(w, bool)  # multiplied at all: with a weight of 0, or one that rounds to it
        touch[o, np.minimum(i0 + 1, n - 1)] = True
        touch[o, np.where(f == 0, np.maximum(i0 - 1, 0), i0)] = True
        zero[o, np.minimum(i0 + 1, n - 1)] = f == 0
        return w, touch, zero

    (wy, ty, zy), (wx, tx, zx) = weights(Hh), weights(W)
    _, _, view = FMT[dtype]
    L = abi.lib()

    def reach(a, b, at):                             # which results an element set at `at` reaches through a and b
        m = np.zeros((a.shape[1], b.shape[1]))
        m[at] = 1
        return a @ m @ b.T > 0

    for at in [(Hh - 1, W - 1), (Hh - 1, 2), (2, W - 1), (2, 3)]:
        x = _q(H.normal(1, shape), dtype)
        x[:, :, at[0], at[1]] = bad
        dx_ = _dev(x, dtype)
        y = _dev(np.zeros((N, Cc, Hh * scale, W * scale), np.float32), dtype)
        abi.check(L.ad_upsample_bilinear_fwd(C.byref(view(dx_)), C.byref(view(y)), scale, 0, Hh, 0, H.stream()))
        H.sync()
        got = ~np.isfinite(_host(y, dtype))
        assert np.all(got >= reach(wy, wx, at)) and np.all(got <= reach(ty, tx, at))
        if not np.isnan(bad):                        # the value itself wherever it is not multiplied with 0 as well
            itself = reach(wy, wx, at) & ~zy[:, at[0], None] & ~zx[None, :, at[1]]
            assert np.all(_host(y, dtype)[:, :, itself] == bad)
        oy, ox = at[0] * scale + scale // 2, at[1] * scale + scale // 2
        dy = _q(H.normal(2, (N, Cc, Hh * scale, W * scale)), dtype)
        dy[:, :, oy, ox] = bad
        ddy = _dev(dy, dtype)
        abi.check(L.ad_upsample_bilinear_bwd(C.byref(view(ddy)), C.byref(view(dx_)), scale, 0, Hh, 0, 0, H.stream()))
        H.sync()
        assert np.array_equal(~np.isfinite(_host(dx_, dtype)), np.broadcast_to(reach(wy.T, wx.T, (oy, ox)), shape))


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("layout", [abi.AD_NCHW, abi.AD_NHWC])
@pytest.mark.parametrize("Cc,HW", [(1, 300), (8, 257), (9, 255), (32, 256), (33, 130), (64, 31), (65, 77), (128, 3), (129, 9), (256, 5), (257, 4), (1000, 1)])
def test_ce_class_counts(dtype, layout, Cc, HW):
    import torch
    N = 3
    logits = _q(H.normal(3, (N, Cc, HW), 2.0), dtype)
    label = H.rng(4).integers(0, Cc, (N, HW)).astype(np.uint32)
    dloss = H.uniform(5, (N, HW))
    loss_w = orc.softmax_ce_pixel_fwd(logits, label)[0]
    dlog_w = orc.softmax_ce_pixel_bwd(logits, label, dloss)
    arr = logits if layout == abi.AD_NCHW else np.ascontiguousarray(np.transpose(logits, (0, 2, 1)))
    d = H.dev(arr) if dtype == "f32" else H.dev_bf16(arr)
    dl, ddl = torch.from_numpy(label.view(np.int32)).cuda(), H.dev(dloss)
    loss, dlog = torch.empty((N, HW), device="cuda"), torch.ones_like(d)
    L, dt = abi.lib(), FMT[dtype][0]
    abi.check(L.ad_softmax_ce_pixel_fwd(dt, layout, N, Cc, HW, H.ptr(d), H.ptr(dl), H.ptr(loss), None, H.stream()))
    abi.check(L.ad_softmax_ce_pixel_bwd(dt, layout, N, Cc, HW, H.ptr(d), H.ptr(dl), H.ptr(ddl), H.ptr(dlog), 1, H.stream()))
    H.sync()
    got = H.host(dlog) - 1
    if layout == abi.AD_NHWC:
        got = np.transpose(got, (0, 2, 1))
    assert H.max_rel(H.host(loss), loss_w) < 1e-5
    assert np.max(np.abs(got - dlog_w)) < (2e-6 if dtype == "f32" else 1e-2)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("shape", [(1, 8, 1, 1), (2, 40, 19, 23), (3, 2048, 7, 7), (5, 264, 5, 4)])
def test_global_average_pool(dtype, shape):
    import torch
    N, Cc, Hh, W = shape
    x, dy = _q(H.normal(6, shape), dtype), _q(H.normal(7, (N, Cc, 1, 1)), dtype)
    y_w, dx_w = orc.avgpool2d_fwd(x, (Hh, W), (1, 1)), orc.avgpool2d_bwd(dy, shape, (Hh, W), (1, 1))
    _, _, view = FMT[dtype]
    dx_, ddy = _dev(x, dtype), _dev(dy, dtype)
    y, gx, ga = torch.empty_like(ddy), torch.empty_like(dx_), torch.ones_like(dx_)
    vx, vy, vdy, vgx, vga = view(dx_), view(y), view(ddy), view(gx), view(ga)
    L = abi.lib()
    abi.check(L.ad_avgpool2d_fwd(C.byref(vx), C.byref(vy), Hh, W, 1, 1, H.stream()))
    abi.check(L.ad_avgpool2d_bwd(C.byref(vdy), C.byref(vgx), Hh, W, 1, 1, 0, H.stream()))
    abi.check(L.ad_avgpool2d_bwd(C.byref(vdy), C.byref(vga), Hh, W, 1, 1, 1, H.stream()))
    H.sync()
    tol = 1e-5 if dtype == "f32" else 1e-2
    assert H.max_rel(_host(y, dtype), y_w) < tol
    assert H.max_rel(_host(gx, dtype), dx_w) < tol
    assert H.max_rel(_host(ga, dtype), 1 + dx_w) < tol


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("B,I,O", [(1, 1, 1), (9, 33, 9), (8, 257, 1000), (17, 512, 7)])
def test_linear_groups(dtype, B, I, O):
    import torch
    x, w, b, dy = _q(H.normal(8, (B, I)), dtype), H.normal(9, (O, I), 0.1), H.normal(10, (O,)), _q(H.normal(11, (B, O)), dtype)
    y_w = orc.linear_fwd(x, w, b)
    dx_w, dw_w, db_w = orc.linear_bwd(x, w, dy)
    mk = H.dev if dtype == "f32" else H.dev_bf16
    dx_, ddy, dw_, db_ = mk(x), mk(dy), H.dev(w), H.dev(b)
    y, gx = torch.empty_like(ddy), torch.ones_like(dx_)
    gw, gb = torch.ones(O, I, device="cuda"), torch.ones(O, device="cuda")
    L, dt = abi.lib(), FMT[dtype][0]
    abi.check(L.ad_linear_fwd(dt, B, I, O, H.ptr(dx_), H.ptr(dw_), H.ptr(db_), H.ptr(y), H.stream()))
    abi.check(L.ad_linear_bwd(dt, B, I, O, H.ptr(dx_), H.ptr(dw_), H.ptr(ddy), H.ptr(gx), H.ptr(gw), H.ptr(gb), 1, 1, H.stream()))
    H.sync()
    tol = 2e-5 if dtype == "f32" else 1e-2
    assert H.max_rel(H.host(y), y_w) < tol
    assert H.max_rel(H.host(gx), 1 + dx_w) < tol
    assert H.max_rel(H.host(gw), 1 + dw_w) < 2e-5
    assert H.max_rel(H.host(gb), 1 + db_w) < 2e-5


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("lift", [0, 1])                # bases off by one element: no vectors
@pytest.mark.parametrize("B,I,O", [
    (9, 1030, 17), (2, 1024, 9), (2, 259, 999), (3, 255, 40),      # images in shared memory: past its 1024 features, at the ends of its range
    (600, 510, 10), (593, 512, 32), (600, 510, 33), (600, 512, 128), (600, 512, 129),   # 4, 8 and 16 warps per block of the data gradient
    (70, 257, 9), (65, 64, 2048), (16, 66, 2049), (17, 66, 2048), (4, 70, 513), (5, 70, 513),   # filter gradient by columns or by fours
])
def test_linear_forms(dtype, lift, B, I, O):
    """Each form of the three kernels at the ends of the range that its rule gives it, against 64 bits."""
    import torch
    x, w, b, dy = _q(H.normal(8, (B, I)), dtype), H.normal(9, (O, I), 0.1), H.normal(10, (O,)), _q(H.normal(11, (B, O)), dtype)
    x64, w64, dy64 = x.astype(np.float64), w.astype(np.float64), dy.astype(np.float64)
    dt, td = FMT[dtype][0], torch.float32 if dtype == "f32" else torch.bfloat16

    def put(a, t):
        flat = torch.full((a.size + 4,), 7.0, dtype=t, device="cuda")
        flat[lift:lift + a.size] = torch.from_numpy(np.ascontiguousarray(a)).cuda().to(t).reshape(-1)
        return flat, flat[lift:lift + a.size].view(a.shape)

    (_, tx), (_, tw), (_, tb), (_, tdy) = put(x, td), put(w, torch.float32), put(b, torch.float32), put(dy, td)
    outs = [put(np.ones((B, O), np.float32), td), put(np.ones_like(x), td), put(np.ones_like(w), torch.float32), put(np.ones_like(b), torch.float32)]
    (_, y), (_, gx), (_, gw), (_, gb) = outs
    L = abi.lib()
    eps = 2.0 ** -24
    half = 0.0 if dtype == "f32" else 2.0 ** -8                    # the result's own rounding
    # a sum of n products: chains of at most n / 32 roundings of partial sums, and the sums of the chains
    far = lambda got, want, mag, n, half: np.all(np.abs(H.host(got) - want) <= (n / 32 + 40) * eps * mag + half * np.abs(want) + 1e-6)  # noqa: E731
    abi.check(L.ad_linear_fwd(dt, B, I, O, H.ptr(tx), H.ptr(tw), H.ptr(tb), H.ptr(y), H.stream()))
    for acc in (1, 0):
        abi.check(L.ad_linear_bwd(dt, B, I, O, H.ptr(tx), H.ptr(tw), H.ptr(tdy), H.ptr(gx), H.ptr(gw), H.ptr(gb), acc, acc, H.stream()))
        H.sync()
        assert far(gx, acc + dy64 @ w64, acc + np.abs(dy64) @ np.abs(w64), O, half)
        assert far(gw, acc + dy64.T @ x64, acc + np.abs(dy64).T @ np.abs(x64), 32 * B, 0.0)
        assert far(gb, acc + dy64.sum(0), acc + np.abs(dy64).sum(0), 32 * B, 0.0)
    assert far(y, x64 @ w64.T + b, np.abs(x64) @ np.abs(w64).T + np.abs(b), I, half)
    for flat, t in outs:                                           # nothing beside the results is written
        t.fill_(7.0)
        assert torch.all(flat == 7.0)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("shape,k,s", [
    ((1, 8, 3, 3), (3, 3), (2, 2)), ((2, 16, 33, 35), (3, 3), (2, 2)), ((1, 24, 17, 16), (2, 2), (2, 2)), ((1, 72, 18, 31), (3, 3), (1, 1)),
    ((1, 40, 20, 21), (2, 5), (1, 3)), ((2, 8, 65, 66), (3, 3), (4, 4)), ((1, 8, 40, 70), (7, 9), (2, 2)), ((1, 8, 37, 37), (17, 2), (1, 1)),
])
def test_maxpool_tiles(dtype, shape, k, s):
    import torch
    N, Cc, Hh, W = shape
    x = _q(np.round(H.normal(12, shape) * 2) / 2, dtype)        # many ties
    y_w = orc.maxpool2d_fwd(x, k, s)
    dy = _q(H.normal(13, y_w.shape), dtype)
    dx_w = orc.maxpool2d_bwd(x, dy, k, s)
    _, _, view = FMT[dtype]
    dx_, ddy = _dev(x, dtype), _dev(dy, dtype)
    y, gx, ga = torch.empty_like(ddy), torch.empty_like(dx_), torch.ones_like(dx_)
    vx, vy, vdy, vgx, vga = view(dx_), view(y), view(ddy), view(gx), view(ga)
    L = abi.lib()
    abi.check(L.ad_maxpool2d_fwd(C.byref(vx), C.byref(vy), *k, *s, H.stream()))
    abi.check(L.ad_maxpool2d_bwd(C.byref(vx), C.byref(vdy), C.byref(vgx), *k, *s, 0, H.stream()))
    abi.check(L.ad_maxpool2d_bwd(C.byref(vx), C.byref(vdy), C.byref(vga), *k, *s, 1, H.stream()))
    H.sync()
    assert np.array_equal(_host(y, dtype), y_w)
    tol = 1e-6 if dtype == "f32" else 1e-2
    assert H.max_rel(_host(gx, dtype), dx_w) < tol
    assert H.max_rel(_host(ga, dtype), 1 + dx_w) < tol


@pytest.mark.parametrize("N,Cc,Hh,W,K", [(1, 64, 3, 5, 8), (2, 64, 40, 130, 64), (1, 128, 65, 67, 256), (3, 64, 33, 31, 19), (1, 64, 70, 300, 520)])
def test_bias_gradient(N, Cc, Hh, W, K):
    import torch
    dy = orc.round_bf16(H.uniform(14, (N, K, Hh, W), -0.5, 1.0))
    L = abi.lib()
    a = conv_args(abi.AD_BF16, abi.AD_NHWC, (N, Cc, Hh, W), K, 1, 1, 1, 0)
    x, ddy = torch.zeros(N, Hh, W, Cc, dtype=torch.bfloat16, device="cuda"), H.dev_bf16(orc.nchw_to_nhwc(dy))
    dw, db = torch.empty(K, 1, 1, Cc, device="cuda"), torch.ones(K, device="cuda")
    scratch = torch.zeros(L.ad_conv2d_scratch_bytes(C.byref(a), 2), dtype=torch.uint8, device="cuda")
    a.x, a.y, a.dw, a.db, a.scratch, a.scratch_bytes, a.accumulate = (x.data_ptr(), ddy.data_ptr(), dw.data_ptr(), db.data_ptr(), scratch.data_ptr(),
                                                                     scratch.numel(), 1)
    dw.zero_()
    abi.check(L.ad_conv2d_wgrad(C.byref(a), H.stream()))
    H.sync()
    assert H.max_rel(H.host(db), 1 + dy.astype(np.float64).sum(axis=(0, 2, 3))) < 1e-5
