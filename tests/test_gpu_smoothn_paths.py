"""smoothn's launch rules: the clusters of CTAs that share a pair (their size
follows the number of pairs) and the DCT kernels' ranges of line lengths.

Every pair of a batch has the same result, bit for bit, as alone, whatever
the cluster size; lines around the kernels' limits (90 / 91 and 860 / 861
positions) match SciPy's DCT at a given parameter.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _env():
    import torch

    from openpiv_gpu import _build, _lib

    _build.build()
    torch.cuda.set_device(0)
    return torch, _lib, _lib.load()


def _fields(seed, pairs, m, n):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:m, 0:n]
    u = np.stack([3 * np.sin(x / (5.0 + k % 7)) + rng.normal(0, 0.2, (m, n)) for k in range(pairs)])
    v = np.stack([2 * np.cos(y / (7.0 + k % 5)) + rng.normal(0, 0.2, (m, n)) for k in range(pairs)])
    return u, v


def _smooth(env, u, v, s, mask=None):
    torch, _lib, lib = env
    pairs, m, n = u.shape
    du, dv = torch.as_tensor(u).cuda(), torch.as_tensor(v).cuda()
    p = torch.empty(pairs, dtype=torch.float64, device="cuda")
    dm = None if mask is None else torch.as_tensor(mask.astype(np.uint8)).cuda()
    _lib.check(lib.piv_smoothn(m, n, pairs, du.data_ptr(), dv.data_ptr(), None if dm is None else dm.data_ptr(), s,
                               p.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return du.cpu().numpy(), dv.cpu().numpy(), p.cpu().numpy()


# 152 SMs: clusters of 8 up to 19 pairs, 4 up to 38, 2 up to 76, then one CTA.
@pytest.mark.parametrize("pairs", [2, 19, 20, 39, 77])
@pytest.mark.parametrize("shape,masked", [((31, 33), None), ((17, 22), 0.05), ((17, 22), 0.3)])
def test_result_does_not_depend_on_the_cluster_size(pairs, shape, masked):
    env = _env()
    u, v = _fields(3, pairs, *shape)
    mask = None
    if masked is not None:  # 0.05: the direct GCV score; 0.3: the score that refits the field
        mask = np.random.default_rng(4).random(shape) < masked
        u[:, mask] = np.nan
        v[:, mask] = np.nan
    ub, vb, pb = _smooth(env, u, v, float("nan"), mask)
    assert np.isfinite(ub).all() and np.isfinite(vb).all()
    for k in sorted({0, 1, pairs // 2, pairs - 1}):
        ua, va, pa = _smooth(env, u[k:k + 1], v[k:k + 1], float("nan"), mask)
        np.testing.assert_array_equal(ua[0], ub[k])
        np.testing.assert_array_equal(va[0], vb[k])
        assert pa[0] == pb[k]


@pytest.mark.parametrize("shape", [(90, 91), (91, 90), (92, 253), (5, 860), (861, 4), (3, 861), (2, 2)])
@pytest.mark.parametrize("pairs", [1, 3])
def test_line_lengths_around_the_kernels_limits(shape, pairs):
    from scipy.fft import dctn, idctn

    m, n = shape
    s = 0.7
    u, v = _fields(5, pairs, m, n)
    got = _smooth(_env(), u, v, s)
    lam = 2 * (2 - (np.cos(np.pi * np.arange(m) / m)[:, None] + np.cos(np.pi * np.arange(n) / n)[None, :]))
    # A dot product of L terms c x with |c| <= sqrt(2 / L): at most L 2^-53
    # sum |c x| <= L^1.5 2^-52.5 max |x|, in each of four passes; the
    # double-float products (L <= 90) are within 1e-13 of the largest value.
    length = max(m, n)
    tol = 4 * (length ** 1.5 * 2.0 ** -52.5 + 1e-13) * max(np.abs(u).max(), np.abs(v).max())
    for k in range(pairs):
        for f, g in ((u, got[0]), (v, got[1])):
            ref = idctn(dctn(f[k], norm="ortho") / (1 + s * lam * lam), norm="ortho")
            np.testing.assert_allclose(g[k], ref, rtol=0, atol=tol)


# A pair alone has three shares of outputs or more, and its inputs are scaled
# by a launch of their own; with 40 pairs the only share scales them itself.
@pytest.mark.parametrize("shape", [(92, 91), (91, 92)])
@pytest.mark.parametrize("s", [0.7, float("nan")])
def test_scaling_before_the_inverse_does_not_depend_on_the_shares(shape, s):
    env = _env()
    u, v = _fields(6, 40, *shape)
    ub, vb, pb = _smooth(env, u, v, s)
    for k in (0, 21, 39):
        ua, va, pa = _smooth(env, u[k:k + 1], v[k:k + 1], s)
        np.testing.assert_array_equal(ua[0], ub[k])
        np.testing.assert_array_equal(va[0], vb[k])
        assert pa[0] == pb[k]
