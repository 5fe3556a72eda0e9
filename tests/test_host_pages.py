"""fault_in_pages (csrc/host_pages.h), which pulls into pageable arrays run before their copy: the
array keeps its contents, and its pages are resident afterwards."""
import ctypes
import mmap
import os
import resource
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ellipsesinflows_gb300", "csrc")


@pytest.fixture(scope="module")
def fault_in(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("pages") / "pages.so")
    code = '#include "host_pages.h"\nextern "C" void run(void *p, size_t n) { eif::fault_in_pages(p, n); }\n'
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-I" + CSRC, "-x", "c++", "-", "-o", lib], input=code, text=True,
                   check=True)
    fn = ctypes.CDLL(lib).run
    fn.argtypes, fn.restype = [ctypes.c_void_p, ctypes.c_size_t], None
    return fn


@pytest.mark.parametrize("nbytes", [0, 1, 4095, 4096, 4097, 12288, 100003])
@pytest.mark.parametrize("offset", [0, 8, 4000])
def test_contents_are_kept(fault_in, nbytes, offset):
    a = np.random.default_rng(1).integers(0, 256, offset + nbytes + 64, dtype=np.uint8)
    want = a.copy()
    fault_in(a.ctypes.data + offset, nbytes)
    assert np.array_equal(a, want)


def test_pages_are_resident_afterwards(fault_in):
    size = 1 << 25
    with mmap.mmap(-1, size, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS) as m:
        a = np.frombuffer(m, dtype=np.uint8)
        fault_in(a.ctypes.data, size)
        before = resource.getrusage(resource.RUSAGE_SELF).ru_minflt
        a[:] = 1
        assert resource.getrusage(resource.RUSAGE_SELF).ru_minflt - before < size // mmap.PAGESIZE // 8
        assert a.min() == 1
        del a
