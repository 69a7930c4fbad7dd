"""The bounded wait of the node gathers: a pair of hexes that never arrives
ends the gather with a status, within the limit, and nothing is added from it
on; the device stays usable."""
import ctypes as C
import time

import pytest

from snac_b200.context import load_library

pytestmark = pytest.mark.gpu

OK, ETIMEDOUT = 0, -8
NX, NY, NZ = 3, 2, 3


def selftest(stages, late, limit_ms):
    f = load_library().snac_gpu_selftest_gather
    f.argtypes = [C.c_int, C.c_int, C.c_double, C.POINTER(C.c_int), C.POINTER(C.c_int)]
    f.restype = C.c_int
    status, counts = C.c_int(1), (C.c_int * 3)()
    t = time.perf_counter()
    assert f(stages, late, limit_ms, C.byref(status), counts) == 0
    return status.value, list(counts), time.perf_counter() - t


def hexes_of_pairs(n):
    """terms of all nodes from the first n of the pairs (j-1, k-1), (j, k-1), (j-1, k), (j, k)"""
    return sum(1 for k in range(NZ + 1) for j in range(NY + 1) for i in range(NX + 1) for c in range(n) for s in range(2)
               if 0 <= i - 1 + s < NX and 0 <= j - 1 + (c & 1) < NY and 0 <= k - 1 + (c >> 1) < NZ)


@pytest.mark.parametrize("stages", [1, 2, 4])
def test_nothing_late(stages):
    status, counts, _ = selftest(stages, -1, 5.0)
    assert (status, counts) == (OK, [64, 64, hexes_of_pairs(4)])


@pytest.mark.parametrize("stages", [1, 2, 4])
@pytest.mark.parametrize("late", [0, 1, 2, 3])
def test_a_pair_that_does_not_arrive(stages, late):
    selftest(stages, -1, 5.0)  # loads the kernel
    status, counts, seconds = selftest(stages, late, 20.0)
    assert status == ETIMEDOUT
    assert counts == [0, 0, hexes_of_pairs(late)]
    # the wait, and again the limit for the copies in flight; not once per later pair
    assert 0.02 <= seconds < 0.5
    assert selftest(stages, -1, 5.0)[0] == OK
