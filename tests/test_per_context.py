"""Bookkeeping of the objects kept per context (scratch pools, set-up streams),
with a fake runtime (no GPU)."""

import ctypes
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture
def pools(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    out = str(tmp_path / "libpools.so")
    r = subprocess.run([nvcc, "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                        os.path.join(HERE, "per_context_harness.cu"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(out)


def test_a_pool_per_device_and_its_own_trim(pools):
    pools.fake_fail(1)
    assert pools.pool_get() == 0  # none: tried again at the next call
    pools.fake_fail(0)
    first = pools.pool_get()
    assert first > 0 and pools.pool_get() == first
    pools.fake_device(3)
    other = pools.pool_get()
    assert other not in (0, first) and pools.pool_get() == other
    # A plan of device 0 goes while device 3 is current.
    pools.pool_trim(0)
    assert (pools.fake_trimmed(first), pools.fake_trimmed(other)) == (1, 0)
    pools.fake_device(0)
    pools.pool_trim(3)
    pools.pool_trim(5)  # a device without a pool
    assert (pools.fake_trimmed(first), pools.fake_trimmed(other)) == (1, 1)
    assert pools.pool_get() == first


def test_a_device_reset_ends_its_pool(pools):
    first = pools.pool_get()
    pools.fake_device(1)
    other = pools.pool_get()
    pools.fake_reset(0)
    assert pools.pool_get() == other
    pools.pool_trim(0)  # the old handle is gone with its context
    assert pools.fake_trimmed(first) == 0
    pools.fake_device(0)
    second = pools.pool_get()
    assert second not in (0, first, other) and pools.pool_get() == second
    pools.pool_trim(0)
    assert (pools.fake_trimmed(first), pools.fake_trimmed(second), pools.fake_trimmed(other)) == (0, 1, 0)
    made = {first, other, second}
    for _ in range(100):  # pools without end: none, which sends the call to the device's own pool
        pools.fake_reset(0)
        made.add(pools.pool_get())
    assert 0 in made and len(made) == 64 + 1
