"""Float64 correlation passes with n_fft 2: a float32 map finds the integer
peak, direct float64 sums give the fit's five values, and windows that the
search leaves open take the float64 transforms.

Checked against the float64 maps (piv_correlate_maps, which always take the
float64 transforms): the same integer peaks in every window, and the fit of
the maps' values within their rounding.
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frames(seed, h, w, dtype, kind):
    rng = np.random.default_rng(seed)
    top = 65535 if dtype == "uint16" else 255
    a = rng.integers(0, top + 1, (h, w)).astype(np.float64)
    b = np.roll(a, (1, -2), (0, 1))
    b[: h // 4] = rng.integers(0, top + 1, (h // 4, w))  # windows without a match
    if kind == "ties":
        a[:, : w // 2] = 3  # constant windows
        b[:, : w // 2] = 3
        a[h // 2:, w // 2:] = np.tile(rng.integers(0, top + 1, (4, 4)), (h, w))[: h - h // 2, : w - w // 2]  # periodic
        b[h // 2:, w // 2:] = a[h // 2:, w // 2:]
    if kind == "offset":  # fractions and a large level: float pixels only
        a = 3.0e6 + a / 7.0
        b = 3.0e6 + b / 7.0
    if kind == "tiny":
        a *= 1e-30
        b *= 1e-30
    if kind == "nan":
        a[h // 2, w // 2] = np.nan
        b[0, 0] = np.inf
    return a.astype(dtype), b.astype(dtype)


@pytest.mark.parametrize("ss", [16, 32, 64])
@pytest.mark.parametrize("dtype,kind", [("uint8", "plain"), ("uint8", "ties"), ("uint16", "plain"), ("float32", "plain"),
                                        ("float64", "plain"), ("float64", "ties"), ("float64", "offset"),
                                        ("float64", "tiny"), ("float64", "nan")])
@pytest.mark.parametrize("shape", [(64, 64), (101, 147)])
@pytest.mark.parametrize("masked", [False, True])  # masked passes take the float64 transforms
def test_peaks_and_fits_are_the_float64_maps(ss, dtype, kind, shape, masked):
    import torch

    from openpiv_gpu import _build, _lib
    from openpiv_gpu.gpu_process import PIVFieldGPU

    _build.build()
    torch.cuda.set_device(0)
    lib = _lib.load()
    h, w = max(shape[0], ss), max(shape[1], ss)
    a, b = _frames(ss + w, h, w, dtype, kind)
    geom = PIVFieldGPU((h, w), ss, overlap_ratio=0.75, dtype_f=np.float64).geometry
    m, n, N = geom.m, geom.n, 2 * ss
    # uint16 has no torch type with every operation: bytes are enough here.
    da, db = (torch.as_tensor(np.ascontiguousarray(f).view(np.uint8)).cuda() for f in (a, b))
    pt = _lib.PIXEL[{"uint8": "u8", "uint16": "u16", "float32": "f32", "float64": "f64"}[dtype]]
    mask = np.zeros((m, n), dtype=np.uint8)
    mask[0, 0] = masked
    dm = torch.as_tensor(mask).cuda()
    mask_ptr = dm.data_ptr() if masked else None
    f64 = _lib.DTYPE["float64"]
    stream = torch.cuda.current_stream().cuda_stream
    maps = torch.empty((m, n, N, N), dtype=torch.float64, device="cuda")
    _lib.check(lib.piv_correlate_maps(ctypes.byref(geom), 1, da.data_ptr(), db.data_ptr(), pt, f64, N, 1,
                                      mask_ptr, maps.data_ptr(), _lib.DFT["fft"], stream))
    u = torch.empty((m, n), dtype=torch.float64, device="cuda")
    v = torch.empty_like(u)
    pi = torch.empty((m, n), dtype=torch.int32, device="cuda")
    pj = torch.empty_like(pi)
    _lib.check(lib.piv_correlate(ctypes.byref(geom), 1, da.data_ptr(), db.data_ptr(), pt, f64, N, 1,
                                 _lib.SUBPIXEL["gaussian"], mask_ptr, u.data_ptr(), v.data_ptr(), pi.data_ptr(),
                                 pj.data_ptr(), 0, 2, None, _lib.DFT["fft"], stream))
    u2, v2 = torch.empty_like(u), torch.empty_like(u)  # without peak arrays: the same fields
    _lib.check(lib.piv_correlate(ctypes.byref(geom), 1, da.data_ptr(), db.data_ptr(), pt, f64, N, 1,
                                 _lib.SUBPIXEL["gaussian"], mask_ptr, u2.data_ptr(), v2.data_ptr(), None, None, 0,
                                 2, None, _lib.DFT["fft"], stream))
    maps, u, v, u2, v2, pi, pj = (t.cpu().numpy() for t in (maps, u, v, u2, v2, pi, pj))
    np.testing.assert_array_equal(u, u2)
    np.testing.assert_array_equal(v, v2)
    flat = maps.reshape(m, n, -1)
    at = np.argmax(np.where(np.isnan(flat), np.inf, flat), axis=2)  # a map of NaN: its first NaN, as argmax has it
    np.testing.assert_array_equal(pi * N + pj, at)
    assert not masked or (np.isnan(u[0, 0]) and np.isnan(v[0, 0]))
    for r in range(m):
        for k in range(n):
            if mask[r, k]:
                continue
            i, j = divmod(int(at[r, k]), N)
            ei, ej, tol = float(i), float(j), 0.0
            if 0 < i < N - 1 and 0 < j < N - 1:
                c, d, up, lf, rt = (maps[r, k, i + y, j + x] for y, x in ((0, 0), (-1, 0), (1, 0), (0, -1), (0, 1)))
                # A map value of the float64 transforms is within 6.7 2^-53
                # log2(N^2) |a| |b| per transform of the exact one; |a| |b| is
                # at most the sum of the products, bounded here by the pixel
                # range's.
                s = slice(r * geom.spacing + geom.y_offset, r * geom.spacing + geom.y_offset + ss)
                t = slice(k * geom.spacing + geom.x_offset, k * geom.spacing + geom.x_offset + ss)
                wa, wb = a[s, t].astype(np.float64), b[s, t].astype(np.float64)
                norm = np.linalg.norm(wa - wa.mean()) * np.linalg.norm(wb - wb.mean())
                # and the means are rounded at the pixels' level
                level = np.abs(wa).max() * np.abs(wb).max() * ss * ss
                err = 3 * 6.7 * 2.0 ** -53 * 14 * norm + 2.0 ** -50 * level ** 0.5 * norm ** 0.5
                if np.isnan(err) or min(c, d, up, lf, rt) <= 4 * err:
                    continue  # not a number, or a positivity test within rounding
                lg = np.log([c, d, up, lf, rt])
                dl = err * np.array([1 / x for x in (c, d, up, lf, rt)])
                di, dj = lg[1] - 2 * lg[0] + lg[2] + 1e-7, lg[3] - 2 * lg[0] + lg[4] + 1e-7
                ei += 0.5 * (lg[1] - lg[2]) / di
                ej += 0.5 * (lg[3] - lg[4]) / dj
                e = 2 * dl.sum()
                if e > 0.1 * min(abs(di), abs(dj)):
                    continue
                tol = 4 * e / min(abs(di), abs(dj)) + 1e-13 * N
            assert abs(v[r, k] + ss - ei) <= tol + 1e-12 and abs(u[r, k] + ss - ej) <= tol + 1e-12, (r, k, tol)
