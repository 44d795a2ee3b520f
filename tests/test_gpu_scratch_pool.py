"""Scratch of the stage entry points: calls from several threads, each on a
stream of its own, and calls inside a stream capture give the results of a
call alone."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(torch, _lib, u, v, stream):
    m, n = u.shape
    p = torch.empty(1, dtype=torch.float64, device="cuda")
    _lib.check(_lib.lib().piv_smoothn(m, n, 1, u.data_ptr(), v.data_ptr(), None, 0.8, p.data_ptr(),
                                      stream.cuda_stream))


def test_threads_streams_and_capture():
    import torch

    from openpiv_gpu import _build, _lib

    _build.build()
    torch.cuda.set_device(0)
    rng = np.random.default_rng(1)
    shapes = [(40, 60), (120, 33), (64, 64), (200, 210)]
    src = [tuple(torch.as_tensor(rng.normal(0, 1, s)).cuda() for _ in range(2)) for s in shapes]
    ref = []
    for u, v in src:
        a, b = u.clone(), v.clone()
        _call(torch, _lib, a, b, torch.cuda.current_stream())
        torch.cuda.synchronize()
        ref.append((a, b))
    bad = []

    def work(k):
        try:
            torch.cuda.set_device(0)
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                for r in range(20):
                    a, b = src[k][0].clone(), src[k][1].clone()
                    _call(torch, _lib, a, b, st)
                    if r % 5 == 0:
                        st.synchronize()
                    if not (torch.equal(a, ref[k][0]) and torch.equal(b, ref[k][1])):
                        bad.append((k, r))
        except Exception as e:  # noqa: BLE001 - reported below
            bad.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(shapes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    # In a capture the scratch belongs to the graph.
    st = torch.cuda.Stream()
    a, b = src[0][0].clone(), src[0][1].clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        p = torch.empty(1, dtype=torch.float64, device="cuda")
        _lib.check(_lib.lib().piv_smoothn(*shapes[0], 1, a.data_ptr(), b.data_ptr(), None, 0.8, p.data_ptr(),
                                          torch.cuda.current_stream().cuda_stream))
    a.copy_(src[0][0])
    b.copy_(src[0][1])
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(a, ref[0][0]) and torch.equal(b, ref[0][1])
