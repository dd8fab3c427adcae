"""Which output buffers the library makes resident before a copy into them, on the
CPU: a read-back (on several threads) from 32 MB on, a buffer that is filled
behind the device's work (one thread) from 1 MB on; smaller ones are left alone,
and no value changes."""
import ctypes as C
import mmap

import numpy as np
import pytest

from mnhack8_b200 import _lib

PAGE = 4096


def resident(buf):
    n = len(buf) // PAGE
    vec = (C.c_ubyte * n)()
    addr = C.addressof(C.c_char.from_buffer(buf))
    libc = C.CDLL(None, use_errno=True)
    assert libc.mincore(C.c_void_p(addr), C.c_size_t(len(buf)), vec) == 0
    return sum(v & 1 for v in vec), n


def touch(buf, size, parallel):
    f = getattr(_lib.lib(), "_ZN2hs11touch_pagesEPvmb")
    f.restype, f.argtypes = None, [C.c_void_p, C.c_size_t, C.c_bool]
    f(C.addressof(C.c_char.from_buffer(buf)), size, parallel)


@pytest.mark.parametrize("parallel,mb,touched", [(True, 1, False), (True, 4, False), (True, 31, False), (True, 32, True),
                                                 (True, 40, True), (False, 0.5, False), (False, 1, True), (False, 8, True)])
def test_which_buffers(parallel, mb, touched):
    size = int(mb * (1 << 20))
    buf = mmap.mmap(-1, size + PAGE, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
    if resident(buf)[0]:
        pytest.skip("this kernel reports fresh pages as resident")
    touch(buf, size + 8, parallel)                       # a ragged end
    got = resident(buf)[0]
    assert (got >= size // PAGE) if touched else got == 0
    buf.close()


@pytest.mark.parametrize("parallel", [True, False])
def test_values_stay(parallel):
    a = np.random.default_rng(1).integers(0, 256, 33 << 20, dtype=np.uint8)
    want = a.copy()
    f = getattr(_lib.lib(), "_ZN2hs11touch_pagesEPvmb")
    f.restype, f.argtypes = None, [C.c_void_p, C.c_size_t, C.c_bool]
    f(a.ctypes.data, a.size, parallel)
    assert np.array_equal(a, want)
