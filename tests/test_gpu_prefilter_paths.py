"""The spline prefilter's loads (words of 8-bit frames, single pixels at the
edges, at odd widths and for the other types; 8-bit regions staged as bytes)
around the 64-pixel tiles and their 12-pixel halo.

The loads only move pixels, and a pixel of 0 .. 255 is the same float whatever
its type, so the coefficients of the four types are equal bit for bit. Against
SciPy's filter in float64: the recursions' float32 rounding, 2^-24 of a partial
sum of at most 255 / (1 - |z|) at every step, amplified by 1 / (1 - |z|) per
recursion, twice per axis, and the start 12 samples out (2e-7 per axis), with
the gain 6 per axis: below 255 * 36 * (8 * 2^-24 * 1.4^4 + 4e-7) < 0.03.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1), (3, 5), (64, 64), (76, 76), (65, 88), (152, 153), (140, 140), (200, 204)])
def test_coefficients_of_every_pixel_type(shape):
    import torch
    from scipy.ndimage import spline_filter

    from openpiv_gpu import _build, _lib

    _build.build()
    torch.cuda.set_device(0)
    lib = _lib.load()
    h, w = shape
    frames = np.random.default_rng(h * w).integers(0, 256, (2, h, w))
    stream = torch.cuda.current_stream().cuda_stream
    got = []
    for code, dtype in enumerate((np.uint8, np.uint16, np.float32, np.float64)):
        f = torch.as_tensor(frames.astype(dtype)).cuda()
        c = torch.full((2, h, w), float("nan"), dtype=torch.float32, device="cuda")
        _lib.check(lib.piv_spline_prefilter(h, w, 2, f.data_ptr(), code, c.data_ptr(), stream))
        got.append(c.cpu().numpy())
    for other in got[1:]:
        np.testing.assert_array_equal(got[0], other)
    if min(shape) > 1:
        for k in range(2):
            ref = spline_filter(frames[k].astype(np.float64), order=3, mode="mirror")
            np.testing.assert_allclose(got[0][k], ref, rtol=0, atol=0.03)
