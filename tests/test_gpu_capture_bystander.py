"""Calls of one thread while another one captures in the global mode: giving
back what a graph that is gone has kept must not spoil that capture."""
import gc
import threading
import time

import numpy as np
import pytest

from conftest import from_device, to_device

pytestmark = pytest.mark.gpu


def test_scratch_of_a_gone_graph_is_freed_beside_a_capture(cuda, oracle, t213):
    d1, d2, eb = 300007, 37, 4  # ragged, with a remainder: scratch
    x = oracle.random_bits(d1 * d2, eb, 5)
    want = oracle.gather213(x.view(np.dtype((np.void, eb))), d1, d2, 1).view(np.uint8)
    dev = to_device(cuda, x)
    warm, other = cuda.cuda.Stream(), cuda.cuda.Stream()
    y = cuda.arange(1 << 16, dtype=cuda.float32, device="cuda")
    cuda.cuda.synchronize()
    with cuda.cuda.stream(warm):
        t213.transpose(to_device(cuda, x), d1, d2, 1, elem_bytes=eb)
        g = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(g, stream=warm):
            t213.transpose(dev, d1, d2, 1, elem_bytes=eb)
    cuda.cuda.synchronize()
    g.reset()
    del g
    gc.collect()
    time.sleep(0.5)  # the graph's scratch comes back on a thread of the driver
    errors = []

    def call():
        try:
            t213.transpose(dev, d1, d2, 1, elem_bytes=eb, stream=warm.cuda_stream)
        except Exception as e:
            errors.append(repr(e))

    g2 = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(g2, stream=other, capture_error_mode="global"):
        th = threading.Thread(target=call)
        th.start()
        th.join()
        y.mul_(2)
    g2.replay()
    cuda.cuda.synchronize()
    assert not errors, errors
    assert np.array_equal(from_device(dev), want)
    assert float(y[3]) == 6.0
