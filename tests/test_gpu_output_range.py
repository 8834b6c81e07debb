"""Which outputs the batcher's kernels write in place: only memory that they
can address to its last byte.  The decision alone; nothing is written."""
import ctypes
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _direct(lib, p, n):
    return bool(lib.rte_output_is_direct(p, n, 0))


def test_host_outputs_must_be_page_locked_throughout(lib, cuda):
    import torch
    page = mmap.PAGESIZE
    raw = np.zeros(5 * page, np.uint8)
    base = -(-raw.ctypes.data // page) * page
    assert not _direct(lib, base, 4)
    rt = torch.cuda.cudart()
    assert int(rt.cudaHostRegister(base, 2 * page, 0)) == 0
    try:
        assert _direct(lib, base, 2 * page) and _direct(lib, base + 4, 2 * page - 4)
        assert _direct(lib, base + 2 * page - 4, 4)
        assert not _direct(lib, base, 2 * page + 1)       # one byte past the page-locked part
        assert not _direct(lib, base, 3 * page)
        assert not _direct(lib, base + 2 * page - 4, 8)
        assert not _direct(lib, base + 2, 4)              # a 4-byte store cannot address it
        assert not _direct(lib, base, 0)
    finally:
        assert int(rt.cudaHostUnregister(base)) == 0
    assert not _direct(lib, base, 2 * page)


def test_device_outputs_must_lie_in_one_allocation(lib, cuda):
    cuda.zeros(1, device="cuda")  # the primary context is current
    drv = ctypes.CDLL("libcuda.so.1")
    size = 32 << 20
    ptr = ctypes.c_uint64()
    assert drv.cuMemAlloc_v2(ctypes.byref(ptr), ctypes.c_size_t(size)) == 0
    a = ptr.value
    try:
        assert _direct(lib, a, size) and _direct(lib, a + size - 4, 4)
        assert not _direct(lib, a, size + 4)
        assert not _direct(lib, a + size - 4, 8)
        assert not bool(lib.rte_output_is_direct(a, size, 1))  # another device's kernels
    finally:
        assert drv.cuMemFree_v2(ctypes.c_uint64(a)) == 0
