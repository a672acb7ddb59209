"""3x3 convolutions whose input stays in shared memory for all taps, against
the fp64 reference of test_gpu_nn_conv.py: widths from 1 to 128 (tiles that
cross image rows, end inside the halo columns, or lie beyond the last row),
image heights of one tile and less than a band, channel counts with partial
slices, several output parts, and inputs too wide for shared memory.

Outputs are rounded to bf16 (half an ulp is 2^-9 of the value), sums are fp32:
the tolerance is that of the shape tests."""
import ctypes

import numpy as np
import pytest

from test_gpu_nn_conv import _torch, as64, bf16, ref_conv, view

pytestmark = pytest.mark.gpu

# n, h, w, cin, cout
SHAPES = [
    (1, 1, 128, 16, 16), (2, 3, 128, 32, 32), (1, 9, 128, 96, 32),
    (1, 5, 128, 256, 48), (1, 2, 128, 320, 32),
    (1, 2, 64, 48, 64), (3, 6, 64, 192, 64), (1, 4, 32, 64, 128),
    (2, 36, 32, 384, 128), (2, 8, 16, 128, 256), (40, 24, 16, 256, 256),
    (1, 16, 8, 64, 96), (2, 64, 2, 32, 16), (1, 128, 1, 16, 32),
]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("masked", [False, True])
def test_band_forward(gpu_lib, shape, masked):
    torch = _torch()
    n, h, w, cin, cout = shape
    rng = np.random.default_rng(h * 131 + w * 17 + cin)
    x = bf16(rng.standard_normal((n, h, w, cin))).cuda()
    wt = bf16(rng.standard_normal((cout, 9, cin)) / np.sqrt(9 * cin)).cuda()
    bias = (rng.standard_normal(cout) * 0.1).astype(np.float32)
    bdev = torch.from_numpy(bias).cuda()
    # the output is a channel slice of a wider buffer
    y = torch.zeros((n, h, w, cout + 16), dtype=torch.bfloat16, device="cuda")
    mask = bf16(rng.standard_normal((n, h, w, cout))).cuda()
    mview = view(mask, n, h, w, cout, cout)
    torch.cuda.synchronize()
    rc = gpu_lib.mplbnn_conv_forward(
        ctypes.byref(view(x, n, h, w, cin, cin)), wt.data_ptr(), 9,
        None if masked else bdev.data_ptr(), 0 if masked else 1,
        ctypes.byref(view(y, n, h, w, cout, cout + 16, 8)), 0,
        ctypes.byref(mview) if masked else None, None)
    assert rc == 0, gpu_lib.mplbnn_error().decode()
    ref = ref_conv(as64(x), as64(wt), 9,
                   None if masked else bias.astype(np.float64), not masked,
                   as64(mask) if masked else None)
    y = as64(y)
    scale = np.abs(ref).max()
    assert np.allclose(y[..., 8:8 + cout], ref, rtol=8e-3, atol=1e-3 * scale)
    assert not y[..., :8].any() and not y[..., 8 + cout:].any()


# n, h, w, cout, cin: rows a band, output slices and groups, partial slices
WGRAD_SHAPES = [
    (1, 1, 128, 16, 16), (2, 3, 128, 32, 32), (1, 9, 128, 32, 96),
    (3, 5, 128, 160, 32), (1, 2, 64, 64, 48), (3, 6, 64, 64, 192),
    (1, 4, 32, 128, 64), (2, 36, 32, 128, 160), (9, 16, 16, 256, 128),
    (40, 24, 16, 96, 256), (1, 16, 8, 96, 64), (2, 64, 2, 16, 32),
    (1, 128, 1, 32, 16),
]


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("shape", WGRAD_SHAPES)
def test_band_wgrad(gpu_lib, shape, shift):
    """Sums of fp32 products of bf16 values over up to 15,360 pixels: rtol
    1e-3 plus 1e-4 of the largest, as the shape tests' weight gradients; added
    to what dw holds."""
    from test_gpu_nn_conv import ref_wgrad
    torch = _torch()
    n, h, w, cout, cin = shape
    rng = np.random.default_rng(h * 131 + w * 17 + cin)
    # slices of wider buffers, whose other channels must not enter
    x = bf16(rng.standard_normal((n, h, w, cin + 16))).cuda()
    dy = bf16(rng.standard_normal((n, h, w, cout + 8))).cuda()
    before = rng.standard_normal((cout, 9, cin)).astype(np.float32)
    # added by bulk reductions, one atomic per lane off 16-byte alignment; what
    # lies around it stays
    mem = torch.full((before.size + 8,), 7.0, device="cuda")
    dw = mem[4 + shift:4 + shift + before.size].view(before.shape)
    dw.copy_(torch.from_numpy(before))
    torch.cuda.synchronize()
    rc = gpu_lib.mplbnn_conv_wgrad(
        ctypes.byref(view(dy, n, h, w, cout, cout + 8, 8)),
        ctypes.byref(view(x, n, h, w, cin, cin + 16, 8)), 9, dw.data_ptr(),
        None)
    assert rc == 0, gpu_lib.mplbnn_error().decode()
    ref = ref_wgrad(as64(dy)[..., 8:8 + cout], as64(x)[..., 8:8 + cin], 9)
    got = dw.cpu().numpy().astype(np.float64) - before
    scale = np.abs(ref).max()
    assert np.allclose(got, ref, rtol=1e-3, atol=1e-4 * scale + 1e-6)
    assert (mem[:4 + shift] == 7).all() and (mem[4 + shift + before.size:] == 7).all()
