"""Descriptors that t213_batch_create refuses, on the host, before it plans or
allocates anything: data that is not aligned to its element size, NULL data,
volumes past 64 bits and plan kinds that have no name, as the plain call refuses
them.  The kernels access whole
elements, so such a tensor must never reach one."""
import ctypes

import pytest

BASE = 1 << 20


def _create(t213, *descs):
    arr = (t213._lib.TensorDesc * len(descs))(*[t213._lib.TensorDesc(*d) for d in descs])
    h = ctypes.c_void_p(0)
    return t213.lib().t213_batch_create(arr, len(descs), ctypes.byref(h)), h.value


@pytest.mark.parametrize("eb", (2, 4, 8, 16))
def test_misaligned_data_is_refused(t213, eb):
    status, handle = _create(t213, (BASE + eb // 2, 33, 17, 3, eb, 0))
    assert status == 1 and not handle
    assert b"aligned" in t213.lib().t213_last_error()


def test_one_bad_descriptor_refuses_the_batch(t213):
    ok = [(BASE + (i << 20), 64, 48, 2, 4, 0) for i in range(4)]
    for bad in ((BASE + 2, 64, 48, 2, 4, 0), (0, 64, 48, 2, 4, 0), (BASE, 1 << 31, 1 << 31, 4, 8, 0)):
        assert _create(t213, *ok, bad) == (1, None)


@pytest.mark.parametrize("kind", (-20, -4, -2, -1, 9, 10, 99))
def test_kinds_without_a_name_are_refused(t213, kind):
    """The planner's internal kinds are no plan of a caller's."""
    assert _create(t213, (BASE, 64, 48, 2, 4, kind)) == (1, None)
    assert b"plan" in t213.lib().t213_last_error()
    buf, n = ctypes.create_string_buffer(256), ctypes.c_int32(0)
    assert t213.lib().t213_plan_describe(64, 48, 2, 4, kind, 0, buf, 256) == 1
    assert t213.lib().t213_plan_launches(64, 48, 2, 4, kind, 0, ctypes.byref(n)) == 1
