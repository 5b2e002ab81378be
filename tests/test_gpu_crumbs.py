"""Many small slices in runs (k_crumbs): slices of the smallest sides, of one
run, runs with remainders, every element size and base offset, the joined steps
of a permutation, the named directions and the batched form.  Bit-exact against
the oracle, guard bytes on both sides."""
import numpy as np
import pytest

from conftest import from_device, to_device

SHAPES = [(2, 2, 297), (3, 3, 4099), (4, 4, 20000), (5, 7, 1001), (2, 100, 1500), (64, 3, 999), (9, 13, 640), (16, 16, 777)]


def test_plan_choice(t213):
    assert t213.describe(4, 4, 100000, 4).startswith("crumbs")
    assert not t213.describe(4, 4, 16, 4).startswith("crumbs")
    assert not t213.describe(100, 100, 100000, 4).startswith("crumbs")


def _place(oracle, count, eb, off, seed):
    x = oracle.random_bits(count, eb, seed)
    guard = 64 + off * eb
    host = np.full(guard + x.nbytes + 64, 0x5A, np.uint8)
    host[guard:guard + x.nbytes] = x.view(np.uint8)
    return x, host, guard


def _check(dev, guard, want):
    got = from_device(dev)
    n = want.size
    assert np.array_equal(got[guard:guard + n], want)
    assert (got[:guard] == 0x5A).all() and (got[guard + n:] == 0x5A).all()


@pytest.mark.gpu
@pytest.mark.parametrize("off", (0, 1, 3))
@pytest.mark.parametrize("eb", (1, 2, 4, 8, 16))
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_small_slices(cuda, oracle, t213, shape, eb, off):
    d1, d2, d3 = shape
    x, host, guard = _place(oracle, d1 * d2 * d3, eb, off, d1 + d2)
    want = oracle.gather213(x.view(np.dtype((np.void, eb))), d1, d2, d3).view(np.uint8)
    for call in (lambda v: t213.transpose(v, d1, d2, d3, elem_bytes=eb),
                 lambda v: t213.c2r_transpose(v, d1, d2, d3, elem_bytes=eb),
                 lambda v: t213.r2c_transpose(v, d2, d1, d3, elem_bytes=eb)):
        dev = to_device(cuda, host)
        call(dev[guard:guard + x.nbytes])
        cuda.cuda.synchronize()
        _check(dev, guard, want)


@pytest.mark.gpu
@pytest.mark.parametrize("off", (0, 1))
@pytest.mark.parametrize("eb", (1, 2, 4, 8, 16))
@pytest.mark.parametrize("dims", [(2, 2, 2, 3000), (3, 5, 4, 777), (7, 2, 9, 1031)], ids=lambda s: "x".join(map(str, s)))
def test_joined_steps(cuda, oracle, t213, dims, eb, off):
    x, host, guard = _place(oracle, int(np.prod(dims)), eb, off, sum(dims))
    want = oracle.seq_tt(x.view(np.dtype((np.void, eb))), list(dims), [2, 1, 0, 3]).view(np.uint8)
    dev = to_device(cuda, host)
    t213.permute(dev[guard:guard + x.nbytes], dims, (2, 1, 0, 3), elem_bytes=eb)
    cuda.cuda.synchronize()
    _check(dev, guard, want)


@pytest.mark.gpu
def test_in_a_batch(cuda, oracle, t213):
    specs = [(4, 4, 50000, 4), (3, 3, 1000, 2), (500, 300, 4, 4), (64, 48, 8, 8), (5, 2, 400, 16)]
    xs = [oracle.random_bits(a * b * c, eb, i) for i, (a, b, c, eb) in enumerate(specs)]
    want = [oracle.gather213(x.view(np.dtype((np.void, s[3]))), *s[:3]).view(np.uint8) for x, s in zip(xs, specs)]
    dev = [to_device(cuda, x) for x in xs]
    B = t213.Batch([(d, *s) for d, s in zip(dev, specs)])
    try:
        B.execute(cuda.cuda.Stream())
        cuda.cuda.synchronize()
        for d, w in zip(dev, want):
            assert np.array_equal(from_device(d), w)
    finally:
        B.close()
