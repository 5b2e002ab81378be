"""Scratch and cycle tables of captured calls belong to the graph: the stream's
workspace may move and the plan may leave the cache before a replay.
Bit-exact against the oracle."""
import numpy as np
import pytest

from conftest import from_device, to_device

pytestmark = pytest.mark.gpu

# rows and columns cut, with and without a remainder
SHAPES = [(6002, 4000, 4), (4000, 6002, 4), (4099, 4101, 2)]


def _case(oracle, d1, d2, eb, seed):
    x = oracle.random_bits(d1 * d2, eb, seed)
    return x, oracle.gather213(x.view(np.dtype((np.void, eb))), d1, d2, 1).view(np.uint8)


def test_replay_after_the_caches_are_released(cuda, oracle, t213):
    cases = [_case(oracle, d1, d2, eb, 11 + i) for i, (d1, d2, eb) in enumerate(SHAPES)]
    dev = [to_device(cuda, x) for x, _ in cases]
    st = cuda.cuda.Stream()
    with cuda.cuda.stream(st):
        for (d1, d2, eb), (x, _) in zip(SHAPES, cases):  # tables on the device
            t213.transpose(to_device(cuda, x), d1, d2, 1, elem_bytes=eb)
        g = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(g, stream=st):
            for (d1, d2, eb), d in zip(SHAPES, dev):
                t213.transpose(d, d1, d2, 1, elem_bytes=eb)
    cuda.cuda.synchronize()
    t213.release_cache()
    with cuda.cuda.stream(st):
        d1, d2, eb = 9001, 7003, 4  # the stream's workspace anew, larger
        t213.transpose(cuda.zeros(d1 * d2, dtype=cuda.float32, device="cuda"), d1, d2, 1, elem_bytes=eb)
        g.replay()
    cuda.cuda.synchronize()
    for d, (_, want) in zip(dev, cases):
        assert np.array_equal(from_device(d), want)
    assert t213.device_status() == 0
    del g


def test_batch_replay_after_the_workspace_moved(cuda, oracle, t213):
    cases = [_case(oracle, d1, d2, eb, 21 + i) for i, (d1, d2, eb) in enumerate(SHAPES)]
    dev = [to_device(cuda, x) for x, _ in cases]
    B = t213.Batch([(d, d1, d2, 1, eb) for d, (d1, d2, eb) in zip(dev, SHAPES)])
    st = cuda.cuda.Stream()
    try:
        B.execute(st)
        assert B.status(st) == 0
        for d, (x, want) in zip(dev, cases):
            assert np.array_equal(from_device(d), want)
            d.copy_(cuda.from_numpy(x.view(np.uint8).reshape(-1)).view(d.dtype))
        cuda.cuda.synchronize()
        t213.release_cache()
        B.execute(st)  # the captured graph
        assert B.status(st) == 0
        for d, (_, want) in zip(dev, cases):
            assert np.array_equal(from_device(d), want)
    finally:
        B.close()
