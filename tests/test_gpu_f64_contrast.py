"""Float64 correlation passes whose two frames differ in contrast: the peak of
every window is the largest value of its float64 correlation.

The oracle transforms the two windows apart (numpy, float64). The device's
float64 transforms take both windows in one complex transform, so a value of
theirs is within 3 x 6.7 2^-53 log2(N^2) (|a|^2 + |b|^2) / 2 of the exact one
(Higham, Accuracy and Stability of Numerical Algorithms, section 24.1); two
values closer than twice that may change places.
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frames(seed, size, kind):
    rng = np.random.default_rng(seed)
    a, b = rng.random((size, size)), rng.random((size, size))  # no match: close runners-up
    b[size // 2:] = np.roll(a, (1, -2), (0, 1))[size // 2:] + 0.5 * b[size // 2:]
    if kind == "counts":  # 16-bit: rare single counts against saturated spots
        a, b = rng.random((size, size)) < 0.05, 65535 * (rng.random((size, size)) < 0.3)
        return a.astype(np.uint16), b.astype(np.uint16)
    if kind == "flat":  # 16-bit: a nearly constant frame
        a = 30000 + (rng.random((size, size)) < 0.02)
        return a.astype(np.uint16), (65535 * b / b.max()).astype(np.uint16)
    scale, dtype = kind
    return a.astype(dtype), (b * scale).astype(dtype)


@pytest.mark.parametrize("ss", [16, 32, 64])
@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("kind", ["counts", "flat", (1.0, "float64"), (65535.0, "float64"), (1e6, "float64"),
                                  (1e-6, "float64"), (2.0 ** 20, "float64"), (2.0 ** 32, "float64"),
                                  (1e6, "float32"), (2.0 ** -20, "float32")], ids=str)
def test_peaks_at_unequal_contrast(ss, swap, kind):
    import torch

    from openpiv_gpu import _build, _lib
    from openpiv_gpu.gpu_process import PIVFieldGPU

    _build.build()
    torch.cuda.set_device(0)
    lib = _lib.load()
    size, N = 256, 2 * ss
    a, b = _frames(ss, size, kind)
    if swap:
        a, b = b, a
    geom = PIVFieldGPU((size, size), ss, overlap_ratio=0.75, dtype_f=np.float64).geometry
    m, n = geom.m, geom.n
    da, db = (torch.as_tensor(np.ascontiguousarray(f).view(np.uint8)).cuda() for f in (a, b))
    pt = _lib.PIXEL[{"uint16": "u16", "float32": "f32", "float64": "f64"}[a.dtype.name]]
    u = torch.empty((m, n), dtype=torch.float64, device="cuda")
    v = torch.empty_like(u)
    pi = torch.empty((m, n), dtype=torch.int32, device="cuda")
    pj = torch.empty_like(pi)
    _lib.check(lib.piv_correlate(ctypes.byref(geom), 1, da.data_ptr(), db.data_ptr(), pt, _lib.DTYPE["float64"], N, 1,
                                 _lib.SUBPIXEL["gaussian"], None, u.data_ptr(), v.data_ptr(), pi.data_ptr(),
                                 pj.data_ptr(), 0, 2, None, _lib.DFT["fft"], torch.cuda.current_stream().cuda_stream))
    pi, pj = pi.cpu().numpy(), pj.cpu().numpy()

    def windows(f):
        w = np.lib.stride_tricks.sliding_window_view(f.astype(np.float64), (ss, ss))
        w = w[geom.y_offset::geom.spacing, geom.x_offset::geom.spacing][:m, :n]
        return w - w.mean(axis=(2, 3), keepdims=True)

    wa, wb = windows(a), windows(b)
    c = np.fft.irfft2(np.conj(np.fft.rfft2(wa, (N, N))) * np.fft.rfft2(wb, (N, N)), (N, N))
    c = np.fft.fftshift(c, axes=(2, 3))
    c[:, :, 0, :] = c[:, :, :, 0] = 0.0  # no overlap
    err = 3 * 6.7 * 2.0 ** -53 * 2 * np.log2(N) * 0.5 * ((wa ** 2).sum(axis=(2, 3)) + (wb ** 2).sum(axis=(2, 3)))
    at = np.take_along_axis(c.reshape(m, n, -1), (pi * N + pj)[..., None].astype(np.int64), axis=2)[..., 0]
    short = c.max(axis=(2, 3)) - at
    bad = short > 2 * err
    assert not bad.any(), (int(bad.sum()), bad.size, float((short / err).max()))
