"""Element-per-thread pooling and upsampling just below 2^32 elements: the grid's last step passes what 32 bits count."""
import ctypes as C

import pytest

from arraydiff_cuda_b200 import abi
from tests import helpers as H

pytestmark = pytest.mark.gpu

SIDE = 65535                       # squared: 2^32 - 131071, and the grid steps by 148 x 16 x 256


def _map(side, fill=None):
    import torch
    t = torch.empty((1, 1, side, side), dtype=torch.bfloat16, device="cuda")
    return t.uniform_(-1, 1) if fill is None else t.fill_(fill)


def test_average_pool():
    import torch
    L, s = abi.lib(), H.stream()
    x, y = _map(SIDE), _map(SIDE, 9.0)
    abi.check(L.ad_avgpool2d_fwd(C.byref(H.view_nchw(x)), C.byref(H.view_nchw(y)), 1, 1, 1, 1, s))
    H.sync()
    assert torch.equal(x, y)
    dy = _map(SIDE // 2)
    abi.check(L.ad_avgpool2d_bwd(C.byref(H.view_nchw(dy)), C.byref(H.view_nchw(y)), 2, 2, 2, 2, 0, s))
    H.sync()
    want = dy * 0.25               # exact
    for i in (0, 1):
        for j in (0, 1):
            assert torch.equal(y[:, :, i:SIDE - 1:2, j:SIDE - 1:2], want)
    assert torch.count_nonzero(y[:, :, SIDE - 1]) == 0 and torch.count_nonzero(y[..., SIDE - 1]) == 0


def test_upsampling():
    """Scale 1 copies in both directions; the low-resolution view skips every other element, as the row kernels do not take."""
    import torch
    L, s = abi.lib(), H.stream()
    low, high = torch.empty((1, 1, SIDE, 2 * SIDE), dtype=torch.bfloat16, device="cuda")[..., ::2], _map(SIDE, 9.0)
    for r in range(0, SIDE, 4096):
        low[:, :, r:r + 4096].uniform_(-1, 1)
    abi.check(L.ad_upsample_bilinear_fwd(C.byref(H.view_nchw(low)), C.byref(H.view_nchw(high)), 1, 0, SIDE, 0, s))
    H.sync()
    assert all(torch.equal(low[:, :, r:r + 4096], high[:, :, r:r + 4096]) for r in range(0, SIDE, 4096))
    low.fill_(9.0)
    abi.check(L.ad_upsample_bilinear_bwd(C.byref(H.view_nchw(high)), C.byref(H.view_nchw(low)), 1, 0, SIDE, 0, 0, s))
    H.sync()
    assert all(torch.equal(low[:, :, r:r + 4096], high[:, :, r:r + 4096]) for r in range(0, SIDE, 4096))
