"""The bounded waits of the one-pass kernels, made to run out: the barrier of a
grid team (with and without tensor memory, one team and several), the barrier
of a batch's rounds and the persistent kernel's dependency waits.  Each launch
comes back on its own after the few milliseconds it was given, reports
T213_ERR_TIMEOUT once, has written nothing past its barrier, and the next call
on the same stream, which uses the same barrier word, is exact."""
import time

import numpy as np
import pytest

from conftest import from_device, to_device

pytestmark = pytest.mark.gpu

T213_ERR_TIMEOUT = 5
# several teams, one team over tensor memory, vector form with two tiles a CTA, one slice
SLICES = [(1000, 999, 6, 4), (3001, 2000, 3, 4), (1024, 1536, 6, 4), (3000, 1999, 1, 4), (2053, 4099, 2, 2)]


def _case(oracle, d1, d2, d3, eb, seed):
    x = oracle.random_bits(d1 * d2 * d3, eb, seed)
    return x, oracle.gather213(x.view(np.dtype((np.void, eb))), d1, d2, d3).view(np.uint8)


@pytest.mark.parametrize("shape", SLICES, ids=lambda s: "x".join(map(str, s)))
def test_team_barrier_runs_out(cuda, oracle, t213, shape):
    L = t213.lib()
    d1, d2, d3, eb = shape
    assert "slice(grid" in t213.describe(*shape), t213.describe(*shape)
    x, want = _case(oracle, *shape, 3)
    dev = to_device(cuda, x)
    st = cuda.cuda.Stream()
    cuda.cuda.synchronize()
    for _ in range(2):
        t0 = time.perf_counter()
        rc = L.t213_slice_debug_stall(dev.data_ptr(), d1, d2, d3, eb, 3_000_000, st.cuda_stream)
        assert rc == 0, L.t213_last_error().decode()
        assert t213.device_status(st) == T213_ERR_TIMEOUT
        assert time.perf_counter() - t0 < 1.0  # the limit given, not the default 2 s
        assert t213.device_status(st) == 0
        assert np.array_equal(from_device(dev), x.view(np.uint8).reshape(-1))
    t213.transpose(dev, d1, d2, d3, elem_bytes=eb, stream=st)
    st.synchronize()
    assert np.array_equal(from_device(dev), want)
    assert t213.device_status(st) == 0


def test_slices_without_such_a_barrier_are_refused(cuda, t213):
    x = cuda.zeros(64 * 48, device="cuda")
    assert t213.lib().t213_slice_debug_stall(x.data_ptr(), 64, 48, 1, 4, 1_000_000, 0) == 2
    assert t213.lib().t213_slice_debug_stall(x.data_ptr(), 64, 48, 1, 4, 0, 0) == 1


@pytest.mark.parametrize("plan", ("auto", "c2r"))
def test_batch_waits_run_out(cuda, oracle, t213, plan):
    """Rounds (automatic plans) and the persistent kernel (forced ones)."""
    L = t213.lib()
    shapes = [(700, 300, 2, 4), (601, 203, 2, 8), (97, 71, 3, 16), (1001, 499, 2, 2), (1500, 1301, 1, 4), (900, 1100, 4, 4)]
    cases = [_case(oracle, *s, 30 + i) for i, s in enumerate(shapes)]
    dev = [to_device(cuda, x) for x, _ in cases]
    tensors = [(d, *s, plan) for d, s in zip(dev, shapes)]
    st = cuda.cuda.Stream()
    b = t213.Batch(tensors)
    try:
        assert ("rounds: 0 of" in b.describe()) == (plan == "c2r"), b.describe()
        b.execute(st)
        assert b.status(st) == 0
        for d, (x, want) in zip(dev, cases):
            assert np.array_equal(from_device(d), want)
            d.copy_(cuda.from_numpy(x.view(np.uint8).reshape(-1)))
        cuda.cuda.synchronize()
        assert L.t213_batch_debug_stall(b._h, 3_000_000, -1) == 0, L.t213_last_error().decode()
        t0 = time.perf_counter()
        b.execute(st)
        assert b.status(st) == T213_ERR_TIMEOUT
        assert time.perf_counter() - t0 < 1.0
        assert b.status(st) == 0
    finally:
        b.close()
    for d, (x, _) in zip(dev, cases):
        d.copy_(cuda.from_numpy(x.view(np.uint8).reshape(-1)))
    cuda.cuda.synchronize()
    b = t213.Batch(tensors)
    try:
        b.execute(st)
        assert b.status(st) == 0
        for d, (_, want) in zip(dev, cases):
            assert np.array_equal(from_device(d), want)
    finally:
        b.close()
