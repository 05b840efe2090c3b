"""The look at a caller's output array before a kernel writes it (sg_populate of the library): memory
that can be written, memory that can only be read, and addresses of which the system knows nothing."""
import ctypes as C
import mmap
import platform

import pytest

from surfacegrowthconsole_gb300 import _lib as L

PAGE = mmap.PAGESIZE
ANON, READ, WRITE = mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS, mmap.PROT_READ, mmap.PROT_WRITE

pytestmark = pytest.mark.skipif(
    platform.system() != "Linux" or tuple(int(x) for x in platform.release().split("-")[0].split(".")[:2]) < (5, 14),
    reason="the system cannot make pages present")


@pytest.fixture
def pages():
    libc = C.CDLL(None)
    libc.mmap.restype, libc.mmap.argtypes = C.c_void_p, [C.c_void_p, C.c_size_t, C.c_int, C.c_int, C.c_int, C.c_long]
    libc.munmap.argtypes, libc.mprotect.argtypes = [C.c_void_p, C.c_size_t], [C.c_void_p, C.c_size_t, C.c_int]
    at = libc.mmap(None, 4 * PAGE, READ | WRITE, ANON, -1, 0)
    yield libc, at
    libc.munmap(at, 4 * PAGE)


def populate(address, size):
    f = L.lib()._Z11sg_populatePvm
    f.restype, f.argtypes = C.c_int, [C.c_void_p, C.c_size_t]
    return f(address, size)


def test_writable_memory(pages):
    _, at = pages
    for first, size in ((0, 4 * PAGE), (5, 7), (PAGE - 1, 2), (4 * PAGE - 1, 1), (0, 0)):
        assert populate(at + first, size) == 1
    assert populate(None, 100) == 1  # an array that is not asked for


def test_memory_that_can_only_be_read(pages):
    libc, at = pages
    assert libc.mprotect(at + PAGE, PAGE, READ) == 0
    assert populate(at + PAGE, 1) == -1
    assert populate(at, 4 * PAGE) == -1       # one page of several
    assert populate(at + 2 * PAGE, PAGE) == 1  # the pages around it
    assert populate(at, PAGE) == 1


def test_memory_that_is_not_known(pages):
    libc, at = pages
    assert libc.munmap(at + 2 * PAGE, PAGE) == 0
    assert populate(at + PAGE, 2 * PAGE) == 0
    assert populate(at, 2 * PAGE) == 1
