"""The batched form's rounds (k_hold_rounds): tensors of every element size,
odd sides, bases off a 16-byte boundary, many small slices, slices of more
than half a round and tensors too large for one, beside tensors of a forced
plan; on a side stream (captured, replayed) and on the default stream.
Bit-exact against the oracle, no byte outside the tensors written."""
import numpy as np
import pytest

from conftest import from_device, to_device

pytestmark = pytest.mark.gpu

# (d1, d2, d3, element bytes, base offset past a 16-byte boundary, plan)
SPECS = [(64, 48, 30, 4, 0, "auto"), (63, 47, 9, 4, 4, "auto"), (333, 777, 2, 1, 3, "auto"), (257, 129, 3, 2, 2, "auto"),
         (256, 128, 3, 2, 0, "auto"), (100, 37, 5, 8, 8, "auto"), (45, 600, 1, 16, 0, "auto"), (2, 30001, 1, 4, 0, "auto"),
         (30001, 2, 2, 2, 0, "auto"), (1001, 1003, 2, 4, 0, "auto"), (1500, 1301, 2, 4, 4, "auto"),
         (1024, 768, 2, 4, 0, "auto"), (2000, 1999, 1, 4, 0, "auto"), (300, 200, 2, 4, 0, "c2r"),
         (256, 192, 1, 8, 0, "blocks"), (1, 1000, 2, 4, 0, "auto"), (3001, 3000, 1, 4, 0, "auto"), (5, 5, 0, 4, 0, "auto")]


def _place(oracle):
    guard, offs, pos = 64, [], 64
    for d1, d2, d3, eb, off, _ in SPECS:
        pos = (pos + 15) // 16 * 16 + off
        offs.append(pos)
        pos += d1 * d2 * d3 * eb + guard
    host = np.full(pos + 16, 0xC3, np.uint8)
    want = host.copy()
    for i, ((d1, d2, d3, eb, _, _), o) in enumerate(zip(SPECS, offs)):
        x = oracle.random_bits(d1 * d2 * d3, eb, 300 + i)
        host[o:o + x.nbytes] = x.view(np.uint8)
        want[o:o + x.nbytes] = oracle.gather213(x.view(np.dtype((np.void, eb))), d1, d2, d3).view(np.uint8)
    return host, want, offs


@pytest.mark.parametrize("side", (True, False), ids=("side stream", "default stream"))
def test_rounds_match_the_oracle(cuda, oracle, t213, side):
    host, want, offs = _place(oracle)
    dev = to_device(cuda, host)
    base = dev.data_ptr()
    assert base % 16 == 0
    B = t213.Batch([(base + o, d1, d2, d3, eb, plan) for (d1, d2, d3, eb, _, plan), o in zip(SPECS, offs)])
    try:
        assert "rounds: 0 of" not in B.describe(), B.describe()
        st = cuda.cuda.Stream() if side else 0
        for _ in range(2):  # the second execute replays the captured graph
            dev.copy_(cuda.from_numpy(host))
            cuda.cuda.synchronize()
            B.execute(st)
            assert B.status(st) == 0
            got = from_device(dev)
            bad = np.flatnonzero(got != want)
            assert bad.size == 0, f"{bad.size} bytes differ, first at byte {bad[0]}"
    finally:
        B.close()
