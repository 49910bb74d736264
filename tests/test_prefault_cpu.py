"""Population of result arrays ahead of a device copy (CPU): fresh pages are faulted in,
pages that are there already cost no thread, contents stay."""
import ctypes as C
import mmap

import numpy as np
import pytest

MB = 1 << 20


def prefault(lib, maps):
    f = lib._ZN2gt8prefaultEPKPdim   # gt::prefault(double* const*, int, size_t): not part of the C-ABI
    f.restype = C.c_size_t
    addr = (C.c_void_p * len(maps))(*(m.ctypes.data for m in maps))
    return f(addr, C.c_int(len(maps)), C.c_size_t(maps[0].nbytes))


def arrays(n, mb):
    return [np.frombuffer(mmap.mmap(-1, mb * MB, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS), np.uint8)
            for _ in range(n)]


@pytest.mark.parametrize("n,mb", [(3, 17), (1, 64), (3, 16)])
def test_only_missing_pages_are_populated(lib, n, mb):
    fresh = arrays(n, mb)
    if prefault(lib, fresh) == 0:
        pytest.skip("this kernel has no MADV_POPULATE_WRITE")
    assert prefault(lib, fresh) == 0             # present now
    written = arrays(n, mb)
    for i, a in enumerate(written):
        a[:] = i + 1
    assert prefault(lib, written) == 0           # present by use
    assert all((a == i + 1).all() for i, a in enumerate(written))
    half = arrays(n, mb)
    half[0][:] = 7
    assert prefault(lib, half) == sum(a.nbytes for a in half[1:])
    assert (half[0] == 7).all() and not any(a.any() for a in half[1:])


def test_small_results_are_left_alone(lib):
    assert prefault(lib, arrays(3, 8)) == 0
