"""Results of a plan run in memory that is not the plan's device's: such
outputs (another GPU's memory, pinned host memory) are copied to, as a kernel of
the plan's device may have no access to them."""

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
UNREGISTERED, HOST, DEVICE, MANAGED = 0, 1, 2, 3  # cudaMemoryType


def test_only_own_device_memory_is_stored_to(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    out = str(tmp_path / "librule.so")
    r = subprocess.run([nvcc, "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                        os.path.join(HERE, "result_memory_harness.cu"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rule = ctypes.CDLL(out).memory_of_device
    for device in (0, 1, 3):
        for at in (0, 1, 3):
            assert rule(DEVICE, at, device) == int(at == device)
            for kind in (UNREGISTERED, HOST, MANAGED):
                assert rule(kind, at, device) == 0


@pytest.mark.gpu
def test_pinned_outputs_are_copied_to():
    import torch

    from openpiv_gpu import _build, _lib
    from openpiv_gpu.gpu_process import PIVGPU

    _build.build()
    torch.cuda.set_device(0)
    lib = _lib.lib()
    rng = np.random.default_rng(5)
    shape = (192, 224)
    a = rng.integers(0, 256, shape).astype(np.uint8)
    fa, fb = (torch.as_tensor(x)[None].cuda() for x in (a, np.roll(a, (1, 2), (0, 1))))
    proc = PIVGPU(shape, min_search_size=16, search_size_iters=(1, 1), overlap_ratio=0.5, n_fft=2, median_tol=2)
    m, n = proc.piv_fields[-1].field_shape
    plan = proc._plan(_lib.PIXEL["u8"], 1)
    st = torch.cuda.Stream()
    results, nodes = [], []
    for pinned in (False, True):
        kw = dict(pin_memory=True) if pinned else dict(device="cuda")
        u, v = (torch.zeros((m, n), dtype=torch.float64, **kw) for _ in range(2))
        val, out = (torch.zeros((m, n), dtype=torch.uint8, **kw) for _ in range(2))
        ptrs = [t.data_ptr() for t in (u, v, val, out)]
        torch.cuda.synchronize()
        _lib.check(lib.piv_plan_run(plan, 1, fa.data_ptr(), fb.data_ptr(), 0, *ptrs, 0, st.cuda_stream))
        st.synchronize()
        results.append([t.cpu().numpy().copy() for t in (u, v, val, out)])
        count = ctypes.c_int()
        _lib.check(lib.piv_plan_graph_capture(plan, 1, fa.data_ptr(), fb.data_ptr(), *ptrs, ctypes.byref(count),
                                              st.cuda_stream))
        nodes.append(count.value)
    for x, y in zip(*results):
        np.testing.assert_array_equal(x, y)
    assert nodes[1] == nodes[0] - 1  # copies in the place of the result kernel
