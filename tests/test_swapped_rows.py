"""Two steps of a rank-N permutation in one pass (launch_slice with swapped
rows): [h2][h1][g1] -> [g1][h1][h2] per slice.  The row order on the CPU, the
kernel against the oracle's seq_tt on the GPU at the edges of its forms."""
import numpy as np
import pytest

from conftest import from_device, to_device


@pytest.mark.parametrize("g1,h1,h2", [(2, 2, 2), (3, 5, 7), (7, 2, 9), (5, 8, 3), (4, 1, 6), (4, 6, 1)])
def test_row_order_equals_two_steps(g1, h1, h2):
    x = np.arange(h2 * h1 * g1).reshape(h2 * h1, g1)
    first = x.T.reshape(g1, h2, h1)  # the slice transposed
    two = first.transpose(0, 2, 1).reshape(g1, h1 * h2)  # then the axes that now come first
    # the kernel's address of output row s: s * seg + (s / h2) * rest, in elements
    seg, rest = h1 * g1, g1 - h1 * h2 * g1
    at = [s * seg + s // h2 * rest for s in range(h1 * h2)]
    one = np.stack([x.reshape(-1)[a:a + g1] for a in at], axis=1)
    assert np.array_equal(one, two)


# dims fastest first, perm in the reference's convention; one CTA, a cluster,
# the whole chip with one and several slices, narrow and wide rows, a unit
# axis, three steps of which the last two join, and steps that do not join
CASES = [((4, 3, 2), (2, 1, 0)), ((100, 60, 48), (2, 1, 0)), ((33, 7, 129, 5), (2, 1, 0, 3)),
         ((16, 300, 211), (2, 1, 0)), ((1000, 31, 33), (2, 1, 0)), ((301, 401, 29, 3), (2, 1, 0, 3)),
         ((20, 1, 30, 17), (3, 2, 1, 0)), ((12, 25, 24, 30), (3, 2, 1, 0)), ((40, 9, 11, 13), (1, 3, 0, 2)),
         ((7, 500, 3, 40), (2, 3, 1, 0)), ((24, 10, 6, 5000), (2, 1, 0, 3))]


@pytest.mark.gpu
@pytest.mark.parametrize("off", (0, 1), ids=("aligned", "offset"))
@pytest.mark.parametrize("eb", (1, 2, 4, 8, 16))
@pytest.mark.parametrize("dims,perm", CASES, ids=lambda v: "x".join(map(str, v)))
def test_permute_in_one_pass(cuda, oracle, t213, dims, perm, eb, off):
    vol = int(np.prod(dims))
    x = oracle.random_bits(vol, eb, sum(dims))
    want = oracle.seq_tt(x.view(np.dtype((np.void, eb))), list(dims), list(perm)).view(np.uint8)
    guard = 64 + off * eb
    host = np.full(guard + x.nbytes + 64, 0xA5, np.uint8)
    host[guard:guard + x.nbytes] = x.view(np.uint8)
    dev = to_device(cuda, host)
    t213.permute(dev[guard:guard + x.nbytes], dims, perm, elem_bytes=eb)
    cuda.cuda.synchronize()
    got = from_device(dev)
    assert np.array_equal(got[guard:guard + x.nbytes], want)
    assert (got[:guard] == 0xA5).all() and (got[guard + x.nbytes:] == 0xA5).all()
    assert t213.device_status() == 0
