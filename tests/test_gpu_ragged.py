"""The ragged band plan (csrc/k_walk.cuh and the band forms of csrc/k_hold.cuh)
of slices larger than the chip's shared memory: both orientations, with and
without a remainder, pitches and bases off a 16-byte boundary, every element
size, several slices, offsets past 4 GB, and a first call inside a capture.
Bit-exact."""
import numpy as np
import pytest

from conftest import from_device, to_device

pytestmark = pytest.mark.gpu

CASES = [
    # (d1, d2, d3, element bytes, base offset)
    (300007, 37, 1, 4, 0),     # odd pitch, remainder columns
    (37, 300007, 1, 4, 4),     # remainder rows, packed narrow band rows
    (86400, 120, 1, 4, 0),     # aligned, no remainder
    (120, 86400, 1, 4, 8),
    (20006, 1000, 2, 4, 4),    # pitch of 8 mod 16, two slices
    (1000, 20006, 2, 4, 0),
    (50003, 101, 1, 8, 8),
    (101, 50003, 1, 8, 0),
    (70001, 37, 1, 16, 0),
    (37, 70001, 1, 16, 0),
    (30011, 1201, 1, 2, 2),
    (1201, 30011, 1, 2, 0),
    (30012, 1200, 1, 2, 0),
    (9001, 4803, 1, 1, 1),
    (4803, 9001, 1, 1, 3),
    (13000003, 3, 1, 1, 0),
    (3, 13000003, 1, 1, 0),
]


@pytest.mark.parametrize("case", CASES, ids=lambda s: "x".join(map(str, s)))
def test_ragged_bands(cuda, oracle, t213, case):
    d1, d2, d3, eb, offset = case
    assert t213.describe(d1, d2, d3, eb).startswith("ragged"), t213.describe(d1, d2, d3, eb)
    x = oracle.random_bits(d1 * d2 * d3, eb, d1 + d2)
    want = oracle.gather213(x.view(np.dtype((np.void, eb))), d1, d2, d3).view(np.uint8)
    guard = np.full(offset + 32, 0x3C, np.uint8)
    dev = to_device(cuda, np.concatenate([guard, x.view(np.uint8), guard[:32]]))
    view = dev[guard.size:guard.size + x.nbytes]
    for _ in range(2):  # the second call reuses the table and the workspace
        view.copy_(cuda.from_numpy(x.view(np.uint8)))
        t213.transpose(view, d1, d2, d3, elem_bytes=eb)
        cuda.cuda.synchronize()
        got = from_device(view)
        bad = np.flatnonzero(got != want)
        assert bad.size == 0, f"{case}: {bad.size} bytes differ, first at byte {bad[0]}"
    assert (from_device(dev[:guard.size]) == 0x3C).all(), "bytes before the tensor were written"
    assert (from_device(dev[guard.size + x.nbytes:]) == 0x3C).all(), "bytes after the tensor were written"
    assert t213.device_status() == 0


@pytest.mark.parametrize("shape", [(200002, 6000, 1, 4), (6000, 200002, 1, 4)], ids=lambda s: "x".join(map(str, s)))
def test_ragged_bands_past_4_gb(cuda, t213, shape):
    d1, d2, d3, eb = shape
    assert t213.describe(*shape).startswith("ragged")
    gen = cuda.Generator(device="cuda").manual_seed(1)
    x = cuda.empty(d1 * d2 * d3, dtype=cuda.int32, device="cuda").random_(generator=gen)
    want = x.view(d3, d2, d1).transpose(1, 2).contiguous().view(-1)
    t213.transpose(x, d1, d2, d3)
    assert cuda.equal(x, want)


def test_first_call_inside_a_capture(cuda, oracle, t213):
    """Neither the cycle table nor the workspace can be allocated there: the
    call takes a plan that needs neither."""
    d1, d2, eb = 6002, 4000, 4
    assert t213.describe(d1, d2, 1, eb).startswith("ragged")
    x = oracle.random_bits(d1 * d2, eb, 3)
    want = oracle.gather213(x.view(np.dtype((np.void, eb))), d1, d2, 1).view(np.uint8)
    dev = to_device(cuda, x)
    st = cuda.cuda.Stream()
    cuda.cuda.synchronize()
    t213.release_cache()
    with cuda.cuda.stream(st):
        g = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(g, stream=st):
            t213.transpose(dev, d1, d2, 1, elem_bytes=eb)
        g.replay()
    cuda.cuda.synchronize()
    assert np.array_equal(from_device(dev), want)
