"""Creating a plan neither waits for work that the caller has queued nor holds
it up, and what it puts into device memory is complete when it returns."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _processor(shape, masked):
    from openpiv_gpu.gpu_process import PIVGPU

    mask = None
    if masked:
        mask = np.zeros(shape, dtype=np.int32)
        mask[:60, :60] = 1
    return PIVGPU(shape, min_search_size=16, search_size_iters=(1, 1), overlap_ratio=0.5, n_fft=2, median_tol=2,
                  mask=mask)


@pytest.mark.parametrize("masked", [False, True])
def test_creation_beside_queued_work(masked):
    import torch

    from openpiv_gpu import _build, _lib

    _build.build()
    torch.cuda.set_device(0)
    shape = (256, 320)
    rng = np.random.default_rng(3)
    a = rng.integers(0, 256, shape).astype(np.uint8)
    b = np.roll(a, (2, -1), (0, 1))
    ta, tb = torch.as_tensor(a)[None].cuda(), torch.as_tensor(b)[None].cuda()
    u8 = _lib.PIXEL["u8"]
    ref = _processor(shape, masked)  # also loads the kernels that a creation launches
    uv = [t.clone() for t in ref.run_batch(ta, tb)]
    proc = _processor(shape, masked)
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    torch.cuda._sleep(1 << 30)  # about half a second on the legacy stream
    done.record()
    proc._plan(u8, 1)
    assert not done.query(), "the creation waited for the caller's work"
    with torch.cuda.stream(torch.cuda.Stream()):  # does not wait for the legacy stream's work
        out = proc.run_batch(ta, tb)
    torch.cuda.synchronize()
    for x, y in zip(uv, out):
        np.testing.assert_array_equal(x.cpu().numpy(), y.cpu().numpy())
