"""The routes of a batch's small slices (the rounds, the persistent kernel as
one band a slice, the tensor's own plan): batches that take each of them and
mixtures, at odd and aligned sides and every element size, plain and replayed.
Bit-exact against the oracle, no byte outside the tensors written."""
import re

import numpy as np
import pytest

from conftest import from_device, to_device

pytestmark = pytest.mark.gpu

# name, (d1, d2, d3, element bytes) and how many of it, tensors expected in
# (the persistent kernel, their own plans, the rounds)
BATCHES = [
    ("bands of many slices", [((48, 60, 300, 4), 6)], (6, 0, 0)),
    ("a few KB", [((32, 24, 1, 8), 4)], (4, 0, 0)),
    ("bytes", [((48, 32, 3, 1), 5)], (5, 0, 0)),
    ("past the size of a batch", [((48, 60, 4000, 4), 2)], (0, 2, 0)),
    ("tiny slices", [((4, 4, 1000, 4), 3), ((16, 16, 30000, 8), 1)], (0, 4, 0)),
    ("one tensor", [((512, 384, 2, 4), 1)], (0, 0, 1)),
    ("beside larger slices", [((512, 384, 2, 4), 2), ((96, 70, 3, 16), 2), ((33, 47, 5, 2), 1)], None),
    ("all three", [((512, 384, 2, 4), 2), ((48, 60, 300, 4), 16), ((4, 4, 1000, 4), 2), ((201, 77, 9, 1), 1)], None),
]


def _counts(desc):
    g = re.search(r"persistent kernel: (\d+) tensors.*graph nodes: (\d+) tensors.*rounds: \d+ of (\d+) tensors", desc)
    return tuple(int(v) for v in g.groups())


@pytest.mark.parametrize("name,specs,routes", BATCHES, ids=[b[0] for b in BATCHES])
def test_routes(cuda, oracle, t213, name, specs, routes):
    shapes = [s for s, n in specs for _ in range(n)]
    offs, pos = [], 64
    for d1, d2, d3, eb in shapes:
        offs.append(pos)
        pos = (pos + d1 * d2 * d3 * eb + 64 + 15) // 16 * 16
    host = np.full(pos + 16, 0x69, np.uint8)
    want = host.copy()
    for i, ((d1, d2, d3, eb), o) in enumerate(zip(shapes, offs)):
        x = oracle.random_bits(d1 * d2 * d3, eb, 500 + i)
        host[o:o + x.nbytes] = x.view(np.uint8)
        want[o:o + x.nbytes] = oracle.gather213(x.view(np.dtype((np.void, eb))), d1, d2, d3).view(np.uint8)
    dev = to_device(cuda, host)
    b = t213.Batch([(dev.data_ptr() + o, *s) for o, s in zip(offs, shapes)])
    try:
        got = _counts(b.describe())
        assert sum(got) == len(shapes)
        if routes:
            assert got == routes, b.describe()
        else:
            assert got[2] > 0, b.describe()
        st = cuda.cuda.Stream()
        for _ in range(2):
            dev.copy_(cuda.from_numpy(host))
            cuda.cuda.synchronize()
            b.execute(st)
            assert b.status(st) == 0
            bad = np.flatnonzero(from_device(dev) != want)
            assert bad.size == 0, f"{bad.size} bytes differ, first at byte {bad[0]}"
    finally:
        b.close()
