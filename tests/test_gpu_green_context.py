"""Streams of a green context, which have some of the device's SMs: plans whose
CTAs wait for one another need them all resident, so on such a stream they take
fewer teams or another plan, decided before the tensor is touched.  Bit-exact
against the oracle, plain and captured."""
import numpy as np
import pytest

from conftest import from_device, to_device

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=(16, 96))
def green_stream(request, cuda):
    drv = pytest.importorskip("cuda.bindings.driver")

    def ok(res):
        if int(res[0]) != 0:
            pytest.skip(f"green contexts are not available: {res[0]}")
        return res[1] if len(res) == 2 else res[1:]

    cuda.zeros(1, device="cuda")
    dev = ok(drv.cuDeviceGet(0))
    sm = ok(drv.cuDeviceGetDevResource(dev, drv.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups, _, _ = ok(drv.cuDevSmResourceSplitByCount(1, sm, 0, request.param))
    desc = ok(drv.cuDevResourceGenerateDesc([groups[0]], 1))
    ctx = ok(drv.cuGreenCtxCreate(desc, dev, int(drv.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM)))
    st = ok(drv.cuGreenCtxStreamCreate(ctx, int(drv.CUstream_flags.CU_STREAM_NON_BLOCKING), 0))
    assert groups[0].sm.smCount < 148
    stream = cuda.cuda.ExternalStream(int(st))
    yield stream
    stream.synchronize()
    drv.cuStreamDestroy(st)
    drv.cuGreenCtxDestroy(ctx)


# several grid teams, one with tensor memory, the whole chip; ragged bands both
# ways round, walked first and walked last
CASES = [(1000, 999, 4, 4), (2000, 3001, 3, 4), (3001, 2000, 1, 4), (4099, 2053, 2, 2), (300007, 37, 1, 4),
         (37, 300007, 1, 4), (86400, 120, 1, 4), (120, 86400, 1, 4), (4500, 3000, 1, 4), (64, 48, 5, 4)]


@pytest.mark.parametrize("captured", (False, True), ids=("plain", "captured"))
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c)))
def test_transpose_on_some_sms(cuda, oracle, t213, green_stream, case, captured):
    d1, d2, d3, eb = case
    x = oracle.random_bits(d1 * d2 * d3, eb, d1)
    want = oracle.gather213(x.view(np.dtype((np.void, eb))), d1, d2, d3).view(np.uint8)
    dev = to_device(cuda, x)
    cuda.cuda.synchronize()
    if captured:
        g = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(g, stream=green_stream):
            t213.transpose(dev, d1, d2, d3, elem_bytes=eb, stream=green_stream)
        with cuda.cuda.stream(green_stream):
            g.replay()
    else:
        t213.transpose(dev, d1, d2, d3, elem_bytes=eb, stream=green_stream)
    green_stream.synchronize()
    assert np.array_equal(from_device(dev), want)
    assert t213.device_status() == 0


def test_joined_permutation_steps_on_some_sms(cuda, oracle, t213, green_stream):
    dims, perm = (100, 60, 48, 20), (2, 1, 0, 3)
    x = oracle.random_bits(int(np.prod(dims)), 4, 1)
    want = oracle.seq_tt(x.view(np.dtype((np.void, 4))), list(dims), list(perm)).view(np.uint8)
    dev = to_device(cuda, x)
    cuda.cuda.synchronize()
    t213.permute(dev, dims, perm, elem_bytes=4, stream=green_stream)
    green_stream.synchronize()
    assert np.array_equal(from_device(dev), want)
    assert t213.device_status() == 0


def test_batch_on_some_sms(cuda, oracle, t213, green_stream):
    """Rounds need all SMs: their tensors run their own plans there, and the
    rounds again on a stream that has them all."""
    shapes = [(1000, 999, 4, 4), (257, 129, 3, 2), (512, 384, 5, 4), (45, 600, 1, 16), (2000, 1999, 1, 4), (64, 48, 30, 1)]
    hosts = [oracle.random_bits(d1 * d2 * d3, eb, 70 + i) for i, (d1, d2, d3, eb) in enumerate(shapes)]
    dev = [to_device(cuda, x) for x in hosts]
    b = t213.Batch([(d, *s) for d, s in zip(dev, shapes)])
    assert "rounds: 0 of" not in b.describe()
    try:
        for st in (green_stream, green_stream, cuda.cuda.Stream(), green_stream):
            for d, x in zip(dev, hosts):
                d.copy_(cuda.from_numpy(x.view(np.uint8).reshape(-1)))
            cuda.cuda.synchronize()
            b.execute(st)
            assert b.status(st) == 0
            for d, x, (d1, d2, d3, eb) in zip(dev, hosts, shapes):
                want = oracle.gather213(x.view(np.dtype((np.void, eb))), d1, d2, d3).view(np.uint8)
                assert np.array_equal(from_device(d), want), (d1, d2, d3, eb)
    finally:
        b.close()
