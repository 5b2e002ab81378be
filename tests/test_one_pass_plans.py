"""Geometry of the one-pass and ragged band plans, on the CPU: over random
shapes the tiles of a plan cover the slice, its CTAs hold all tiles, its
shared memory fits an SM, and a ragged plan's parts and remainder make up the
longer side; slices larger than the chip are refused as one-pass plans."""
import math
import random
import re

import pytest

SLICE = re.compile(r"slice\((cta|cluster|grid) tiles=(\d+) of (\d+)x(\d+) per cta=(\d+) ctas=(\d+) teams=(\d+)( vec| tmem)?")
RAGGED = re.compile(r"ragged t=(\d+): (cols|rows)\(q=(\d+) r=(\d+) seg=(\d+)B chunks=\d+ carry=\d+\) ")


def _check_slice(desc, m, n, d3, eb):
    g = SLICE.search(desc)
    assert g, desc
    mode, form = g[1], g[8]
    T, tm, tn, S, ctas, teams = (int(v) for v in g.groups()[1:7])
    assert 1 <= tm <= m and 1 <= tn <= n, desc
    assert math.ceil(m / tm) * math.ceil(n / tn) == T <= ctas * S, desc
    assert mode == ("cta" if ctas == 1 else "cluster" if ctas <= 16 else "grid"), desc
    per_sm, smem = (1, 232448) if form == " tmem" else (2, 233472 // 2 - 1024)
    assert S * tm * tn * eb <= smem, desc  # the padding comes on top, inside the kernel's own limit
    assert 1 <= teams <= d3
    if mode == "grid":
        assert teams * ctas <= per_sm * 148, desc
    if form == " vec":
        assert eb in (2, 4) and n * eb % 16 == 0 and m * eb % 16 == 0 and tm * eb % 16 == 0 and tn * eb % 16 == 0, desc


def _shapes(seed, count):
    rng = random.Random(seed)
    for _ in range(count):
        eb = rng.choice((1, 2, 4, 8, 16))
        size = math.exp(rng.uniform(math.log(100), math.log(6e8))) / eb
        d3 = rng.choice((1, 1, 2, 5, 16, 400))
        area = max(4.0, size / d3)
        a = max(2, int(math.exp(rng.uniform(math.log(2), math.log(area) / 2))))
        b = max(2, int(area / a))
        if rng.random() < 0.4:
            a, b = max(8, a // 8 * 8), max(8, b // 8 * 8)
        yield (a, b, d3, eb) if rng.random() < 0.5 else (b, a, d3, eb)


@pytest.mark.parametrize("seed", range(4))
def test_plans_cover_their_slices(t213, seed):
    kinds = {"slice": 0, "ragged": 0}
    for d1, d2, d3, eb in _shapes(seed, 250):
        desc = t213.describe(d1, d2, d3, eb)
        family = desc.split(" ")[0].rstrip(":")
        if family == "slice":
            _check_slice(desc, d2, d1, d3, eb)
        elif family == "ragged":
            g = RAGGED.match(desc)
            assert g, desc
            t, q, r, seg = int(g[1]), int(g[3]), int(g[4]), int(g[5])
            cols = g[2] == "cols"
            assert q * t + r == (d1 if cols else d2) and 0 <= r and seg == t * eb, desc
            assert d1 * d2 * eb > 24e6, desc
            _check_slice(desc, *((d2, t) if cols else (t, d1)), d3 * q, eb)
        kinds[family] = kinds.get(family, 0) + 1
    assert kinds["slice"] > 20 and kinds["ragged"] > 0, kinds


def test_larger_slices_are_refused(t213):
    with pytest.raises(t213.T213Error) as e:
        t213.describe(6001, 2000, 3, 4, "slice")
    assert e.value.status == 2
