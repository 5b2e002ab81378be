"""A shape's first call inside a stream capture: the cycle table is uploaded
beside the capture, whatever the plan, so that the captured launches find it
at the first replay.  Bit-exact against the oracle."""
import numpy as np
import pytest

from conftest import from_device, to_device

pytestmark = pytest.mark.gpu

# (d1, d2, d3, element bytes, plan): ragged bands whose plan of other families
# is blocks and segment cycles, both ways round; that plan itself; bands
CASES = [(3800, 2600, 1, 8, "auto"), (2600, 3800, 1, 8, "auto"), (4700, 1900, 1, 8, "blocks"),
         (4096, 6000, 1, 4, "bands"), (3, 1 << 18, 2, 4, "bands")]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c)))
def test_first_call_captured(cuda, oracle, t213, case):
    d1, d2, d3, eb, plan = case
    x = oracle.random_bits(d1 * d2 * d3, eb, d1)
    want = oracle.gather213(x.view(np.dtype((np.void, eb))), d1, d2, d3).view(np.uint8)
    dev, src = to_device(cuda, x), to_device(cuda, x)
    st = cuda.cuda.Stream()
    cuda.cuda.synchronize()
    t213.release_cache()
    with cuda.cuda.stream(st):
        g = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(g, stream=st):
            t213.transpose_with_plan(dev, d1, d2, d3, plan, elem_bytes=eb)
        for _ in range(2):
            dev.copy_(src)
            g.replay()
            st.synchronize()
            assert np.array_equal(from_device(dev), want)
        dev.copy_(src)
        t213.transpose_with_plan(dev, d1, d2, d3, plan, elem_bytes=eb)  # and outside, on the same table
        st.synchronize()
    assert np.array_equal(from_device(dev), want)
    assert t213.device_status() == 0


def test_captured_permutation_keeps_its_table(cuda, oracle, t213):
    """A permutation's segment step reads its cycle table at every replay: the
    graph keeps it when 256 later tables have pushed it out of the cache."""
    dims, perm = (128, 40, 60, 3), (0, 2, 1, 3)  # segments of 512 bytes
    x = oracle.random_bits(int(np.prod(dims)), 4, 9)
    want = oracle.seq_tt(x.view(np.dtype((np.void, 4))), list(dims), list(perm)).view(np.uint8)
    dev = to_device(cuda, x)
    st = cuda.cuda.Stream()
    cuda.cuda.synchronize()
    with cuda.cuda.stream(st):
        g = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(g, stream=st):
            t213.permute(dev, dims, perm, elem_bytes=4)
    for k in range(300):
        assert "segment_cycles" in t213.describe(16, 8 * (k + 100), 1, 4, "bands", 8)
    t213.release_cache()
    filler = [cuda.full((1 << 18,), -1, dtype=cuda.int32, device="cuda") for _ in range(16)]
    with cuda.cuda.stream(st):
        g.replay()
        st.synchronize()
    assert np.array_equal(from_device(dev), want)
    del filler
