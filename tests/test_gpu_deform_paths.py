"""The bilinear deformation of both frames against the general kernel.

With a predictor halved (exactly), deforming one frame by the whole of it samples
the points that deforming both by a half each does, by the general kernel: the
frames are equal bit for bit, for every pixel type, with and without a mask,
around the 256 x 8 blocks and for spacings down to 1.
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,size,spacing", [((40, 255), 16, 8), ((39, 256), 16, 8), ((33, 257), 9, 1),
                                                ((130, 530), 32, 5)])
@pytest.mark.parametrize("pixel", ["u8", "u16", "f32", "f64"])
@pytest.mark.parametrize("masked", [False, True])
def test_both_frames_are_the_general_kernels(shape, size, spacing, pixel, masked):
    import torch

    from openpiv_gpu import _build, _lib

    _build.build()
    torch.cuda.set_device(0)
    lib = _lib.load()
    h, w = shape
    m, n = (h - size) // spacing + 1, (w - size) // spacing + 1
    g = _lib.PivGeometry(height=h, width=w, search_size=size, window_size=size, spacing=spacing, m=m, n=n, x_offset=0,
                         y_offset=0)
    rng = np.random.default_rng(h * w + spacing)
    dtype = {"u8": np.uint8, "u16": np.uint16, "f32": np.float32, "f64": np.float64}[pixel]
    fa, fb = (torch.as_tensor(rng.integers(0, 250, (2, h, w)).astype(dtype)).cuda() for _ in range(2))
    up, vp = (torch.as_tensor(rng.normal(0, 6, (2, m, n))).cuda() for _ in range(2))
    mask = torch.as_tensor((rng.random((h, w)) < 0.1).astype(np.uint8)).cuda() if masked else None
    stream = torch.cuda.current_stream().cuda_stream

    def deform(u, v, par):
        out = [torch.empty((2, h, w), dtype=torch.float32, device="cuda") for _ in range(2)]
        _lib.check(lib.piv_deform(ctypes.byref(g), 2, fa.data_ptr(), fb.data_ptr(), _lib.PIXEL[pixel], u.data_ptr(),
                                  v.data_ptr(), par, 1, None, None, None if mask is None else mask.data_ptr(), 0,
                                  out[0].data_ptr(), out[1].data_ptr(), stream))
        return [o.cpu().numpy() for o in out]

    both = deform(up, vp, 0.5)
    np.testing.assert_array_equal(both[0], deform(up / 2, vp / 2, 0.0)[0])
    np.testing.assert_array_equal(both[1], deform(up / 2, vp / 2, 1.0)[1])
