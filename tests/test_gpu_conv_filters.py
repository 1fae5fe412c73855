"""Filter preparation and the KCRS filter-gradient reduction against plain PyTorch forms of the same data."""
import ctypes as C

import pytest

from arraydiff_cuda_b200 import abi
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes", [
    [(64, 64, 1, 1)], [(19, 64, 1, 1)], [(130, 192, 1, 1)], [(8, 2, 1, 1)],          # 1x1: whole and ragged filter tiles
    [(64, 64, 3, 3)], [(33, 96, 3, 3)], [(7, 5, 3, 3)],                               # 3x3: constant and variable extents
    [(64, 3, 7, 7)], [(5, 9, 2, 5)], [(3, 4, 17, 17)],                                # others; more taps than the tile holds
    [(32 + i, 64, 3, 3) if i % 3 else (3, 2, 17, 18) for i in range(33)],             # more filters than one launch takes
])
@pytest.mark.parametrize("pad_row", [0, 45])
def test_filter_prepare(shapes, pad_row):
    import torch
    items, outs = (abi.FilterItem * len(shapes))(), []
    for n, (K, Cc, kh, kw) in enumerate(shapes):
        w = torch.randn(K, Cc, kh, kw, device="cuda")
        row, Kp = kh * kw * Cc + pad_row, (K + 63) // 64 * 64
        krsc = torch.full((K, row), 3.0, dtype=torch.bfloat16, device="cuda")
        crsk = None if pad_row else torch.full((Cc, kh, kw, Kp), 3.0, dtype=torch.bfloat16, device="cuda")
        items[n] = abi.FilterItem(w.data_ptr(), krsc.data_ptr(), crsk.data_ptr() if crsk is not None else None, row, K, Cc, kh, kw, Kp, 0)
        outs.append((w, krsc, crsk))
    abi.check(abi.lib().ad_filter_prepare(len(shapes), items, H.stream()))
    H.sync()
    for (K, Cc, kh, kw), (w, krsc, crsk) in zip(shapes, outs):
        n = kh * kw * Cc
        assert torch.equal(krsc[:, :n], w.permute(0, 2, 3, 1).reshape(K, n).bfloat16()) and torch.all(krsc[:, n:] == 3.0)
        if crsk is not None:
            assert torch.equal(crsk[..., :K], w.flip(2, 3).permute(1, 2, 3, 0).bfloat16()) and torch.all(crsk[..., K:] == 0)


@pytest.mark.parametrize("K,Cc,k", [
    (64, 64, 2), (40, 128, 3), (19, 64, 9), (8, 64, 10),
    (256, 128, 3), (200, 192, 1), (520, 128, 2), (384, 256, 1)])   # CTA pairs: whole, ragged; an odd number of filter tiles
@pytest.mark.parametrize("accumulate", [0, 1])
def test_filter_gradient_order(K, Cc, k, accumulate):
    """The KRSC form against a double-precision sum; the KCRS form is the KRSC form, turned round, to the bit."""
    import torch
    N, Hh = 2, 24
    L = abi.lib()
    a = abi.Conv2dArgs()
    a.dtype, a.layout = abi.AD_BF16, abi.AD_NHWC
    a.N, a.C, a.H, a.W, a.K, a.kh, a.kw = N, Cc, Hh, Hh, K, k, k
    a.stride_h = a.stride_w = a.dil_h = a.dil_w = 1
    P = Hh - k + 1
    x, dy = (torch.randn(N, n, n, c, device="cuda").bfloat16() for n, c in ((Hh, Cc), (P, K)))
    sb = L.ad_conv2d_scratch_bytes(C.byref(a), 2)
    scratch, status = torch.zeros(sb, dtype=torch.uint8, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    a.x, a.y, a.scratch, a.scratch_bytes, a.accumulate = x.data_ptr(), dy.data_ptr(), scratch.data_ptr(), sb, accumulate
    old = torch.randn(K, k, k, Cc, device="cuda")
    krsc, kcrs = old.clone(), old.permute(0, 3, 1, 2).clone(memory_format=torch.contiguous_format)
    for out, order in ((krsc, 0), (kcrs, 1)):
        a.dw, a.dw_kcrs = out.data_ptr(), order
        abi.check(L.ad_conv2d_wgrad_ex(C.byref(a), H.ptr(status), H.stream()))
    H.sync()
    assert int(status[0]) == 0 and torch.equal(kcrs, krsc.permute(0, 3, 1, 2))
    x, d = x.cpu().double(), dy.cpu().double().reshape(-1, K).T
    want = torch.stack([torch.stack([d @ x[:, r:r + P, s:s + P].reshape(-1, Cc) for s in range(k)], 1) for r in range(k)], 1)
    want += accumulate * old.cpu().double()
    assert (krsc.cpu() - want).abs().max() < 1e-4 * want.abs().max()


@pytest.mark.parametrize("case", [
    # N, C, H, W, K, k, stride, dil, pad, columns
    (2, 64, 15, 21, 64, 3, 2, 1, 1, None), (1, 256, 9, 140, 64, 1, 2, 1, 0, None), (3, 128, 8, 8, 64, 3, 2, 1, 0, (1, 6)),
    (1, 64, 22, 19, 128, 3, 2, 2, 2, None),      # dilation and stride share a factor: half of the classes have no taps
    (1, 64, 20, 23, 64, 3, 3, 1, 1, None),       # nine classes: three launches
    (2, 64, 17, 16, 64, 2, 3, 1, 0, (2, 9)),     # a kernel smaller than the stride
    (1, 64, 23, 26, 64, 5, 4, 3, 4, None), (1, 19, 12, 12, 64, 3, 2, 1, 1, None), (2, 32, 14, 14, 19, 4, 2, 1, 1, None),
    (1, 64, 31, 33, 64, 7, 2, 1, 3, None),
    # more than 128 channels and 8 slabs of 64: CTA pairs
    (2, 256, 17, 19, 512, 1, 2, 1, 0, None),     # three of four classes have no taps
    (1, 200, 15, 22, 128, 3, 2, 1, 1, (2, 17)),  # ragged channels, a range of columns
    (3, 264, 13, 9, 64, 3, 2, 1, 1, None),       # two channel tiles, the second one of 8
    (1, 256, 20, 47, 64, 3, 3, 1, 1, None),      # nine classes
    (1, 130, 11, 12, 64, 3, 2, 1, 1, None),      # scattered stores
])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_strided_data_gradient(case, accumulate):
    import numpy as np
    import torch
    from oracle import orc
    N, Cc, Hh, W, K, k, s, d, pd, cols = case
    P, Q = ((n + 2 * pd - d * (k - 1) - 1) // s + 1 for n in (Hh, W))
    w = orc.round_bf16(H.normal(1, (K, Cc, k, k), float(np.sqrt(2.0 / (k * k * Cc)))))
    dy = orc.round_bf16(H.uniform(2, (N, K, P, Q)))
    want = orc.conv2d_dgrad(dy, w, (N, Cc, Hh, W), (s, s), (d, d), (pd, pd), omp=True)
    L = abi.lib()
    a = abi.Conv2dArgs()
    a.dtype, a.layout = abi.AD_BF16, abi.AD_NHWC
    a.N, a.C, a.H, a.W, a.K, a.kh, a.kw = N, Cc, Hh, W, K, k, k
    a.stride_h = a.stride_w = s
    a.dil_h = a.dil_w = d
    a.pad_h = a.pad_w = pd
    if cols:
        a.dx_col_begin, a.dx_col_count = cols
    tw, tdy = H.dev_bf16(np.ascontiguousarray(np.transpose(w, (0, 2, 3, 1)))), H.dev_bf16(orc.nchw_to_nhwc(dy))
    dx = torch.full((N, Hh, W, Cc), 3.0, dtype=torch.bfloat16, device="cuda")
    sb = L.ad_conv2d_scratch_bytes(C.byref(a), 1)
    scratch = torch.zeros(sb, dtype=torch.uint8, device="cuda")
    a.w, a.y, a.dx, a.scratch, a.scratch_bytes, a.accumulate = tw.data_ptr(), tdy.data_ptr(), dx.data_ptr(), scratch.data_ptr(), sb, accumulate
    abi.check(L.ad_conv2d_dgrad(C.byref(a), H.stream()))
    H.sync()
    assert scratch[:4].view(torch.int32).item() == 0
    lo, n = cols or (0, W)
    got = orc.nhwc_to_nchw(H.host(dx))
    assert H.max_rel(got[..., lo:lo + n] - 3.0 * accumulate, want[..., lo:lo + n]) < 2e-2
    assert np.all(got[..., :lo] == 3.0) and np.all(got[..., lo + n:] == 3.0)


@pytest.mark.parametrize("case", [
    # N, C, H, W, K, k: long contractions and more than 128 output channels run as CTA pairs
    (1, 512, 9, 29, 256, 1), (3, 512, 11, 13, 200, 1),     # an odd number of pixel tiles; ragged channels (scattered stores)
    (2, 128, 21, 20, 264, 3), (1, 1024, 16, 16, 520, 1),   # several channel tiles, the last one ragged
    (1, 512, 8, 16, 256, 1),                               # a single pixel tile: no pair
])
@pytest.mark.parametrize("bias", [0, 1])
def test_forward_pairs(case, bias):
    import torch
    N, Cc, Hh, W, K, k = case
    L = abi.lib()
    a = abi.Conv2dArgs()
    a.dtype, a.layout = abi.AD_BF16, abi.AD_NHWC
    a.N, a.C, a.H, a.W, a.K, a.kh, a.kw = N, Cc, Hh, W, K, k, k
    a.stride_h = a.stride_w = a.dil_h = a.dil_w = 1
    x, w, b = (torch.randn(*n, device="cuda") for n in ((N, Hh, W, Cc), (K, k, k, Cc), (K,)))
    x, w = x.bfloat16(), w.bfloat16()
    y = torch.full((N, Hh - k + 1, W - k + 1, K), 3.0, dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    a.x, a.w, a.y, a.bias = x.data_ptr(), w.data_ptr(), y.data_ptr(), b.data_ptr() if bias else None
    a.scratch, a.scratch_bytes = status.data_ptr(), 16
    abi.check(L.ad_conv2d_fprop(C.byref(a), H.stream()))
    H.sync()
    want = torch.nn.functional.conv2d(x.cpu().float().permute(0, 3, 1, 2), w.cpu().float().permute(0, 3, 1, 2), b.cpu() if bias else None)
    assert int(status[0]) == 0 and (y.cpu().float() - want.permute(0, 2, 3, 1)).abs().max() < 8e-3 * want.abs().max()


@pytest.mark.parametrize("case", [
    # N, C, H, W, K, k: the epilogue's forms (pair, single CTA, one chunk per tile), ragged channels, scattered stores, row kernel
    (2, 512, 15, 29, 256, 1), (2, 128, 9, 21, 520, 1), (1, 64, 20, 17, 264, 3), (3, 64, 7, 9, 128, 1), (2, 128, 13, 11, 64, 1),
    (2, 128, 10, 12, 19, 1), (1, 64, 9, 140, 64, 3),
])
@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("rows", [None, (2, 3)])
def test_forward_with_addend(case, pad, rows):
    """To the bit: the convolution, rounded, plus the addend."""
    import torch
    N, Cc, Hh, W, K, k = case
    L = abi.lib()
    a = abi.Conv2dArgs()
    a.dtype, a.layout = abi.AD_BF16, abi.AD_NHWC
    a.N, a.C, a.H, a.W, a.K, a.kh, a.kw = N, Cc, Hh, W, K, k, k
    a.stride_h = a.stride_w = a.dil_h = a.dil_w = 1
    P, Q = Hh - k + 1, W - k + 1
    x, w, b = (torch.randn(*n, device="cuda") for n in ((N, Hh, W, Cc), (K, k, k, Cc), (K,)))
    x, w = x.bfloat16(), w.bfloat16()
    add = (20 * torch.randn(N, P + 2 * pad, Q + 2 * pad, K, device="cuda")).bfloat16()
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    a.x, a.w, a.bias, a.scratch, a.scratch_bytes = x.data_ptr(), w.data_ptr(), b.data_ptr(), status.data_ptr(), 16
    if rows:
        a.out_row_begin, a.out_row_count = rows
    lo, n = rows or (0, P)
    y0, y1 = (torch.full((N, P, Q, K), 3.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    a.y = y0.data_ptr()
    abi.check(L.ad_conv2d_fprop(C.byref(a), H.stream()))
    a.y = y1.data_ptr()
    abi.check(L.ad_conv2d_fprop_add(C.byref(a), C.byref(H.view_nhwc(add, (pad, P, Q))), H.stream()))
    H.sync()
    y0[:, lo:lo + n] += add[:, pad + lo:pad + lo + n, pad:pad + Q]
    assert int(status[0]) == 0 and torch.equal(y0, y1)


@pytest.mark.parametrize("case", [
    # N, C, H, W, K, k: the sum in the epilogue (pair, single CTA); behind it (row kernel, scattered stores)
    (2, 512, 15, 29, 256, 1), (3, 64, 7, 9, 128, 1), (1, 64, 9, 140, 64, 3), (2, 128, 10, 12, 24, 1),
])
def test_addend_in_the_output_buffer(case):
    """Refused where it shares memory with the rows that are written, in every form alike; fine beside them."""
    import torch
    N, Cc, Hh, W, K, k = case
    L = abi.lib()
    a = abi.Conv2dArgs()
    a.dtype, a.layout = abi.AD_BF16, abi.AD_NHWC
    a.N, a.C, a.H, a.W, a.K, a.kh, a.kw = N, Cc, Hh, W, K, k, k
    a.stride_h = a.stride_w = a.dil_h = a.dil_w = 1
    P, Q = Hh - k + 1, W - k + 1
    x, w = torch.randn(N, Hh, W, Cc, device="cuda").bfloat16(), torch.randn(K, k, k, Cc, device="cuda").bfloat16()
    buf = torch.randn(N, P + 1, 2 * Q, K, device="cuda").bfloat16()   # y: the left half of the first P rows
    before = buf.clone()
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    a.x, a.w, a.scratch, a.scratch_bytes, a.y = x.data_ptr(), w.data_ptr(), status.data_ptr(), 16, buf.data_ptr()
    a.y_pitch, a.y_plane = 2 * Q * K, (P + 1) * 2 * Q * K

    def add(view):
        return L.ad_conv2d_fprop_add(C.byref(a), C.byref(H.view_nhwc(view)), H.stream())

    assert add(buf[:, :P, :Q]) == -1 and add(buf[:, 1:, :Q]) == -1 and add(buf[:, :P, 1:Q + 1]) == -1
    a.out_row_begin, a.out_row_count = 1, 2
    assert add(buf[:, :P, :Q]) == -1
    H.sync()
    assert torch.equal(buf, before)
    a.out_row_count = a.out_row_begin = 0
    abi.check(add(buf[:, 1:, Q:]))
    want = torch.empty((N, P, Q, K), dtype=torch.bfloat16, device="cuda")
    a.y, a.y_pitch, a.y_plane = want.data_ptr(), 0, 0
    abi.check(L.ad_conv2d_fprop(C.byref(a), H.stream()))
    H.sync()
    assert int(status[0]) == 0 and torch.equal(buf[:, :P, :Q], want + before[:, 1:, Q:])
    assert torch.equal(buf[:, :, Q:], before[:, :, Q:]) and torch.equal(buf[:, P], before[:, P])
