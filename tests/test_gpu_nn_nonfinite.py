"""Weight gradients of 3x3 convolutions over an input with an infinity in its
first and in its last column, at every image width: the taps that use the pixel
become infinite, the others stay what they are.  All values are small whole
numbers, so the sums are exact and compared as such."""
import ctypes

import numpy as np
import pytest

from test_gpu_nn_conv import _torch, bf16, view

pytestmark = pytest.mark.gpu


def taps_of(dy, x):
    """dw[n][tap][c] over the pixels that lie in the image, none of the halo."""
    h, w = x.shape[1:3]
    out = np.zeros((dy.shape[3], 9, x.shape[3]))
    for t in range(9):
        dh, dw = t // 3 - 1, t % 3 - 1
        ys, xs = slice(max(0, -dh), h - max(0, dh)), slice(max(0, -dw),
                                                           w - max(0, dw))
        yi, xi = slice(max(0, dh), h - max(0, -dh)), slice(max(0, dw),
                                                           w - max(0, -dw))
        out[:, t] = np.einsum("byxn,byxc->nc", dy[:, ys, xs], x[:, yi, xi])
    return out


@pytest.mark.parametrize("cout", [32, 96])
@pytest.mark.parametrize("w", [1, 2, 4, 8, 16, 32, 64, 128])
def test_infinity_enters_its_taps_only(gpu_lib, w, cout):
    torch = _torch()
    n, h, cin = 2, 2 * 128 // w, 48
    rng = np.random.default_rng(w + cout)
    x = rng.integers(1, 4, (n, h, w, cin)).astype(np.float64)
    dy = rng.integers(1, 4, (n, h, w, cout)).astype(np.float64)
    x[0, h // 2, w - 1, 5] = np.inf
    x[1, h // 2, 0, 37] = np.inf
    ref = taps_of(dy, x)
    xd, dyd = bf16(x).cuda(), bf16(dy).cuda()
    dw = torch.zeros((cout, 9, cin), device="cuda")
    torch.cuda.synchronize()
    rc = gpu_lib.mplbnn_conv_wgrad(
        ctypes.byref(view(dyd, n, h, w, cout, cout)),
        ctypes.byref(view(xd, n, h, w, cin, cin)), 9, dw.data_ptr(), None)
    assert rc == 0, gpu_lib.mplbnn_error().decode()
    assert np.array_equal(dw.cpu().numpy().astype(np.float64), ref)
