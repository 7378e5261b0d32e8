"""CPU test: which problems dpe_ncc_eval_noalloc takes.  The capacity is looked at before the device, and a call
without queries returns right behind it."""
import ctypes as C

import numpy as np
import pytest

import dpe_b200 as D

CAPACITY, RESERVED = 16 << 20, 9472


def _status(n, w, hgt):
    q = D.NCCQuery()
    q.width, q.height, q.num_images = w, hgt, n
    byte = np.zeros(1, np.float32)  # never read
    for i in range(n):
        q.images[i] = byte.ctypes.data
    q.params = D.reference_default_params()
    q.count = 0
    return D.load_library().dpe_ncc_eval_noalloc(C.byref(q), C.c_void_p(byte.ctypes.data), None)


def _bytes(n, w, hgt):
    return n * (((w + 2) * (hgt + 2) * 4 + 255) // 256 * 256)


def _sizes(lo, hi):
    """Problems whose images take more than lo and at most hi bytes."""
    return [(n, w, hgt) for n in (2, 3, 5, 8, 12) for w in range(300, 2000, 7) for hgt in range(200, 1500)
            if lo < _bytes(n, w, hgt) <= hi][:20]


@pytest.mark.parametrize("over", [False, True])
def test_capacity_limit(over):
    free = CAPACITY - RESERVED
    sizes = _sizes(free, free + 2048) if over else _sizes(free - 768, free)
    assert len(sizes) > 3
    for s in sizes:
        assert _status(*s) == (D.ERR_CAPACITY if over else D.OK), s
