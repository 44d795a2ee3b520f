"""The plain form's kernels for n_fft 2 (piv_corr_fft_half.cuh) against the
general kernel of the same radix split, which the autotuner's variants keep:
the same displacements, peaks and near-tie flags, bit for bit.

Pixels are whole numbers whose window sums are exact in float32, so that the
variants' different summation orders of the means cannot differ.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Window size -> a variant of the general kernel with the default's radix split.
SAME_RADIX = {16: 3, 32: 1, 64: 1}


def _frames(seed, h, w, dtype):
    rng = np.random.default_rng(seed)
    a = rng.integers(0, 256, (2, h, w)).astype(dtype)
    b = np.roll(a, (2, -3), (1, 2))
    b[:, : h // 3] = rng.integers(0, 256, (2, h // 3, w))  # windows without a match
    a[1, :, : w // 2] = 7  # constant windows: every map value is a tie
    return a, b


def _run(proc, a, b, variant):
    from openpiv_gpu import _lib

    plan = proc.plan_handle(a, a.shape[0])
    _lib.check(_lib.lib().piv_plan_set_variant(plan, 0, variant))
    u, v = proc.run_batch(a, b, host_out=True)
    ties = proc.near_ties()
    out = [proc.iteration_outputs(k)[0] for k in range(a.shape[0])]
    return [u.copy(), v.copy()], ties, out


@pytest.mark.parametrize("ss", [16, 32, 64])
@pytest.mark.parametrize("dtype", ["uint8", "uint16", "float32"])
@pytest.mark.parametrize("shape", [(64, 64), (97, 211)])
@pytest.mark.parametrize("extra", ["plain", "mask", "s2n", "nan"])
def test_same_bits_as_the_general_kernel(ss, dtype, shape, extra):
    from openpiv_gpu.gpu_process import PIVGPU

    if extra == "nan" and dtype != "float32":
        pytest.skip("whole-number frames hold no NaN")
    h, w = max(shape[0], ss), max(shape[1], ss)
    a, b = _frames(ss + h, h, w, dtype)
    kw = {}
    if extra == "mask":
        mask = np.zeros((h, w), dtype=bool)
        mask[h // 2:, w // 2:] = True
        kw["mask"] = mask
    if extra == "s2n":
        kw["s2n_tol"] = 1.1
    if extra == "nan":
        a[0, h // 2, w // 2] = np.nan
        b[1, 3, 3] = np.inf
    proc = PIVGPU((h, w), ss, overlap_ratio=0.75, dtype_f="float32", dft="fft", **kw)
    new = _run(proc, a, b, 0)
    old = _run(proc, a, b, SAME_RADIX[ss])
    assert new[1] == old[1]
    for x, y in zip(new[0], old[0]):
        np.testing.assert_array_equal(x, y)
    for x, y in zip(new[2], old[2]):
        for key in ("u_corr", "v_corr", "i_peak", "j_peak", "near_tie", "val0") + (("s2n",) if extra == "s2n" else ()):
            np.testing.assert_array_equal(x[key], y[key], err_msg=key)


# The second peak outside a box of half width `size`: boxes that wrap
# around, one row and column left, and nothing left.
@pytest.mark.parametrize("ss", [32, 64])
@pytest.mark.parametrize("size", [1, 7, 31, 32, 63, 64])
def test_second_peak_is_the_general_kernels(ss, size):
    from openpiv_gpu.gpu_process import PIVGPU

    a, b = _frames(ss + size, 3 * ss, 4 * ss, "uint8")
    proc = PIVGPU(a.shape[1:], ss, overlap_ratio=0.5, dtype_f="float32", dft="fft", s2n_tol=1.1, s2n_size=size,
                  s2n_method="peak2peak")
    new = _run(proc, a, b, 0)
    old = _run(proc, a, b, SAME_RADIX[ss])
    for x, y in zip(new[2], old[2]):
        for key in ("i_peak", "j_peak", "s2n", "val0"):
            np.testing.assert_array_equal(x[key], y[key], err_msg=key)
