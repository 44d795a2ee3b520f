"""Spring replacement around its launch rules: up to 2,048 outliers every
outlier is a row of the solve, beyond that only the coupled ones are (up to
2,048 of them; more take the general iteration). Each against SciPy's direct
solution of the same system."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(f, bad):
    from scipy.sparse import lil_matrix
    from scipy.sparse.linalg import spsolve

    m, n = f.shape
    pos = np.argwhere(bad)
    rank = {tuple(p): k for k, p in enumerate(pos)}
    A, b = lil_matrix((len(pos), len(pos))), np.zeros(len(pos))
    for k, (i, j) in enumerate(pos):
        near = [(i + y, j + x) for y, x in ((-1, 0), (0, -1), (0, 1), (1, 0)) if 0 <= i + y < m and 0 <= j + x < n]
        A[k, k] = len(near)
        for q in near:
            if q in rank:
                A[k, rank[q]] = -1.0
            else:
                b[k] += f[q]
    out = f.copy()
    out[bad] = np.atleast_1d(spsolve(A.tocsc(), b))
    return out


@pytest.mark.parametrize("shape,fraction", [((40, 50), 0.001), ((40, 50), 0.05), ((60, 70), 0.45), ((110, 120), 0.15),
                                            ((110, 120), 0.17), ((200, 211), 0.05), ((90, 90), 0.5)])
def test_spring_matches_the_direct_solution(shape, fraction):
    import torch

    from openpiv_gpu import _build
    from openpiv_gpu.gpu_validation import ReplacementGPU

    _build.build()
    torch.cuda.set_device(0)
    rng = np.random.default_rng(int(1000 * fraction) + shape[0])
    y, x = np.mgrid[0:shape[0], 0:shape[1]]
    u, v = 3 * np.sin(x / 9.0) + y / 50.0, 2 * np.cos(y / 7.0)
    bad = rng.random(shape) < fraction
    bad[0, 0] = bad[0, 1] = bad[-1, 3] = True  # a corner and edges, coupled and alone
    rep = ReplacementGPU(shape, method="spring", dtype_f="float64")
    gu, gv = rep(torch.as_tensor(u).cuda(), torch.as_tensor(v).cuda(), val_locations=bad)
    # The iterations stop where the residual's norm is 1e-14 of the right-hand
    # side's; the smallest eigenvalue of the system is above pi^2 / L^2 of its
    # clusters' extent L, at most 40 points at these fractions.
    for g, f in ((gu, u), (gv, v)):
        rhs = 4 * np.abs(f).max() * np.sqrt(bad.sum())
        np.testing.assert_allclose(g.cpu().numpy(), _reference(f, bad), rtol=0, atol=1e-14 * rhs * 40 ** 2 / np.pi ** 2)
