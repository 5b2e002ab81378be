"""The one-pass slice kernel (csrc/k_hold.cuh): every team form (one CTA,
cluster, cooperative grid), every element size, tile remainders both ways,
packed narrow rows, several slices per team, bases off a 16-byte boundary with
guard bytes, captured launches, and concurrent streams.  Bit-exact against the
oracle."""
import numpy as np
import pytest

from conftest import from_device, to_device

pytestmark = pytest.mark.gpu

# (d1, d2, d3): what the shape is there for
SHAPES = [
    (64, 48, 4),       # one CTA per slice, aligned rows
    (63, 47, 5),       # one CTA, odd both ways
    (100, 100, 400),   # more slices than resident teams
    (257, 129, 3),     # cluster, one row and one column past a tile
    (513, 385, 40),    # clusters, several slices each
    (2, 30001, 2),     # packed rows of two elements
    (30001, 3, 2),     # output rows of three elements
    (1001, 1003, 3),   # grid teams for the larger elements
    (1500, 1001, 5),   # grid, two tiles per CTA, several slices per team
    (1024, 1000, 2),   # 16-byte pitch one way only for small elements
]


def _run(cuda, oracle, t213, d1, d2, d3, eb, offset, seed):
    x = oracle.random_bits(d1 * d2 * d3, eb, seed)
    want = oracle.gather213(x.view(np.dtype((np.void, eb))), d1, d2, d3).view(np.uint8)
    guard = np.full(offset + 32, 0x3C, np.uint8)
    dev = to_device(cuda, np.concatenate([guard, x.view(np.uint8), guard[:32]]))
    view = dev[guard.size:guard.size + x.nbytes]
    t213.transpose_with_plan(view, d1, d2, d3, "slice", elem_bytes=eb)
    cuda.cuda.synchronize()
    got = from_device(view)
    bad = np.flatnonzero(got != want)
    assert bad.size == 0, f"{(d1, d2, d3, eb)}: {bad.size} bytes differ, first at byte {bad[0]}"
    assert (from_device(dev[:guard.size]) == 0x3C).all(), "bytes before the tensor were written"
    assert (from_device(dev[guard.size + x.nbytes:]) == 0x3C).all(), "bytes after the tensor were written"
    assert t213.device_status() == 0


@pytest.mark.parametrize("offset", (0, 1, 2, 4, 8))
@pytest.mark.parametrize("eb", (1, 2, 4, 8, 16))
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_slices_in_one_pass(cuda, oracle, t213, shape, eb, offset):
    if offset % eb and not (offset == 0):
        pytest.skip("the base keeps the element alignment")
    _run(cuda, oracle, t213, *shape, eb, offset, seed=sum(shape) + eb + offset)


@pytest.mark.parametrize("shape", [(2000, 3001, 1, 4), (2048, 2040, 1, 4), (1999, 1001, 1, 16), (4099, 2053, 2, 2)],
                         ids=lambda s: "x".join(map(str, s)))
def test_slices_over_the_whole_chip(cuda, oracle, t213, shape):
    assert "slice(grid" in t213.describe(*shape)
    _run(cuda, oracle, t213, *shape, 0, seed=shape[0])


def test_slice_too_large_is_refused(t213):
    with pytest.raises(t213.T213Error) as e:
        t213.describe(4000, 4001, 1, 4, "slice")
    assert e.value.status == 2


def test_captured_launches_and_streams(cuda, oracle, t213):
    """Grid launches replayed from a graph on one stream while plain calls run
    on two others: every tensor exact, the device status clean."""
    d1, d2, eb = 1001, 1003, 4
    x = [oracle.random_bits(d1 * d2, eb, 5 + i) for i in range(6)]
    want = [oracle.gather213(v.view(np.dtype((np.void, eb))), d1, d2, 1).view(np.uint8) for v in x]
    dev = [to_device(cuda, v) for v in x]
    cap = cuda.cuda.Stream()
    side = [cuda.cuda.Stream(), cuda.cuda.Stream()]
    scratch = to_device(cuda, x[0])
    with cuda.cuda.stream(cap):
        t213.transpose_with_plan(scratch, d1, d2, 1, "slice", elem_bytes=eb)
        cap.synchronize()
        g = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(g, stream=cap):
            t213.transpose_with_plan(dev[0], d1, d2, 1, "slice", elem_bytes=eb)
            t213.transpose_with_plan(dev[1], d1, d2, 1, "slice", elem_bytes=eb)
    cuda.cuda.synchronize()
    with cuda.cuda.stream(cap):
        g.replay()
    for i in range(2, 6):
        with cuda.cuda.stream(side[i % 2]):
            t213.transpose_with_plan(dev[i], d1, d2, 1, "slice", elem_bytes=eb)
    cuda.cuda.synchronize()
    for d, w in zip(dev, want):
        assert np.array_equal(from_device(d), w)
    assert t213.device_status() == 0
    del g


@pytest.mark.parametrize("shape", [(3001, 4000, 1, 4), (1000, 999, 2, 8), (9001, 30, 3, 4), (500001, 30, 1, 4)],
                         ids=lambda s: "x".join(map(str, s)))
def test_named_directions(cuda, oracle, t213, shape):
    """The decomposition's entry points over slices that fit the chip and
    slices that do not (those run the named passes)."""
    d1, d2, d3, eb = shape
    x = oracle.random_bits(d1 * d2 * d3, eb, d1)
    want = oracle.gather213(x.view(np.dtype((np.void, eb))), d1, d2, d3).view(np.uint8)
    calls = [lambda v: t213.c2r_transpose(v, d1, d2, d3, elem_bytes=eb),
             lambda v: t213.r2c_transpose(v, d2, d1, d3, elem_bytes=eb)]
    if d2 <= 32:
        calls.append(lambda v: t213.skinny_c2r_transpose(v, d1, d2, d3, elem_bytes=eb))
    for call in calls:
        dev = to_device(cuda, x)
        call(dev)
        cuda.cuda.synchronize()
        assert np.array_equal(from_device(dev), want)


@pytest.mark.parametrize("e", (80, 256, 496))
@pytest.mark.parametrize("dims", [(13, 1000, 2), (300, 7, 5), (33, 31, 40), (600, 80, 2)],
                         ids=lambda s: "x".join(map(str, s)))
def test_wide_elements(cuda, t213, dims, e):
    """Merged leading axes of a rank-N permutation as elements of several
    16-byte words."""
    h, s, b = dims
    g = cuda.Generator(device="cuda").manual_seed(e + h)
    x = cuda.empty(b * s * h * e, dtype=cuda.uint8, device="cuda").random_(0, 256, generator=g)
    want = x.view(b, s, h, e).permute(0, 2, 1, 3).contiguous().view(-1)
    t213.permute(x, [e, h, s, b], [0, 2, 1, 3], elem_bytes=1)
    assert cuda.equal(x, want)
