"""The regrid's weights (integer intervals, quotients by a product and one
correction) and its two forms (source rows staged in shared memory, or read
directly where they are too long): the oracle's float64 interpolation, bit for
bit, for odd spacings and search sizes, points outside the source grid and
fields of one row or column.
"""

import ctypes

import numpy as np
import pytest

from oracle import piv_oracle as po

pytestmark = pytest.mark.gpu


def _grid(spacing, size, offset, length):
    return np.arange(length) * float(spacing) + size / 2.0 + offset


# (search size, spacing, x offset, y offset, m, n) of source and destination.
CASES = [
    ((32, 16, 3, 5, 9, 11), (16, 8, -2, 1, 21, 25)),
    ((33, 7, 0, 0, 12, 14), (15, 3, -9, 40, 31, 37)),
    ((21, 13, 4, 4, 2, 2), (9, 1, -30, -30, 40, 130)),
    ((64, 49, 1, 0, 5, 1400), (32, 17, 0, 2, 8, 4096)),
    ((16, 10, 0, 0, 3, 1030), (16, 10, 0, 0, 3, 1030)),
]


@pytest.mark.parametrize("src,dst", CASES)
@pytest.mark.parametrize("pairs", [1, 17])
def test_regrid_is_the_oracles(src, dst, pairs):
    import torch

    from openpiv_gpu import _build, _lib

    _build.build()
    torch.cuda.set_device(0)
    lib = _lib.load()
    geo = []
    for ss, sp, xo, yo, m, n in (src, dst):
        geo.append(_lib.PivGeometry(height=1, width=1, search_size=ss, window_size=ss, spacing=sp, m=m, n=n, x_offset=xo,
                                    y_offset=yo))
    rng = np.random.default_rng(pairs)
    u, v = rng.normal(0, 3, (2, pairs, src[4], src[5]))
    du, dv = torch.as_tensor(u).cuda(), torch.as_tensor(v).cuda()
    gu = torch.empty((pairs, dst[4], dst[5]), dtype=torch.float64, device="cuda")
    gv = torch.empty_like(gu)
    _lib.check(lib.piv_regrid(ctypes.byref(geo[0]), ctypes.byref(geo[1]), pairs, du.data_ptr(), dv.data_ptr(),
                              gu.data_ptr(), gv.data_ptr(), torch.cuda.current_stream().cuda_stream))
    sy, sx = _grid(src[1], src[0], src[3], src[4]), _grid(src[1], src[0], src[2], src[5])
    y, x = np.meshgrid(_grid(dst[1], dst[0], dst[3], dst[4]), _grid(dst[1], dst[0], dst[2], dst[5]), indexing="ij")
    for k in {0, pairs - 1}:
        np.testing.assert_array_equal(gu[k].cpu().numpy(), po.grid_interp(sy, sx, u[k], y, x))
        np.testing.assert_array_equal(gv[k].cpu().numpy(), po.grid_interp(sy, sx, v[k], y, x))
