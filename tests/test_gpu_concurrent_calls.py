"""Two host threads whose calls keep bytes in a stream's workspace between
launches (a ragged transpose's remainder and carries, a row gather through
scratch, a blocks plan's carries), on one stream and on the threads' own
per-thread default streams (one handle for all of them).  Every result
bit-exact against the oracle."""
import threading

import numpy as np
import pytest

from conftest import from_device, to_device

pytestmark = pytest.mark.gpu

PER_THREAD = 2  # cudaStreamPerThread

# (d1, d2, element bytes, plan): remainder and carries; rows through scratch,
# a larger workspace; carries of small segments
JOBS = [(300007, 37, 4, "auto"), (60001, 401, 4, "c2r"), (5000, 3500, 4, "blocks")]


def _jobs(cuda, oracle, t213):
    assert t213.describe(*JOBS[0][:2], 1, 4).startswith("ragged")
    assert "scratch" in t213.describe(*JOBS[1][:2], 1, 4, "c2r")
    out = []
    for i, (d1, d2, eb, plan) in enumerate(JOBS):
        x = oracle.random_bits(d1 * d2, eb, 60 + i)
        want = oracle.gather213(x.view(np.dtype((np.void, eb))), d1, d2, 1).view(np.uint8)
        out.append((to_device(cuda, x), [to_device(cuda, x) for _ in range(6)], want))
    return out


def _run(cuda, t213, jobs, stream_of):
    """Each thread: its job over six tensors, four times, on stream_of(thread)."""
    bad, errors = [], []
    go = threading.Barrier(len(jobs))

    def work(i):
        try:
            src, bufs, want = jobs[i]
            d1, d2, eb, plan = JOBS[i]
            st = stream_of(i)
            for _ in range(4):
                for b in bufs:
                    b.copy_(src)
                cuda.cuda.synchronize()
                go.wait(60)
                for b in bufs:
                    if plan == "auto":
                        t213.transpose(b, d1, d2, 1, elem_bytes=eb, stream=st)
                    else:
                        t213.transpose_with_plan(b, d1, d2, 1, plan=plan, elem_bytes=eb, stream=st)
                go.wait(60)
                cuda.cuda.synchronize()
                bad.extend(f"{JOBS[i]}: tensor {k}" for k, b in enumerate(bufs) if not np.array_equal(from_device(b), want))
                go.wait(60)
        except Exception as e:  # reported by the test, not lost with the thread
            go.abort()
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors and not bad, (errors, bad)
    assert t213.device_status() == 0


def test_threads_on_one_stream(cuda, oracle, t213):
    st = cuda.cuda.Stream()
    _run(cuda, t213, _jobs(cuda, oracle, t213), lambda i: st)


def test_threads_on_their_per_thread_streams(cuda, oracle, t213):
    _run(cuda, t213, _jobs(cuda, oracle, t213), lambda i: PER_THREAD)


def test_a_new_stream_under_an_old_handle(cuda, oracle, t213):
    """A destroyed stream's last call may still run when its handle, and with it
    the workspace, comes back for a new stream."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    jobs = _jobs(cuda, oracle, t213)
    for rep in range(3):
        (d1, d2, eb, plan), (src, bufs, want) = JOBS[0], jobs[0]
        for b in bufs:
            b.copy_(src)
        cuda.cuda.synchronize()
        handles = []
        for b in bufs:
            err, st = rt.cudaStreamCreateWithFlags(rt.cudaStreamNonBlocking)
            assert int(err) == 0
            handles.append(int(st))
            t213.transpose(b, d1, d2, 1, elem_bytes=eb, stream=int(st))
            assert int(rt.cudaStreamDestroy(st)[0]) == 0
        cuda.cuda.synchronize()
        for b in bufs:
            assert np.array_equal(from_device(b), want), f"handles {handles}"
