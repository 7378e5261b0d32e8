"""CPU test: the Python side sizes pyramid levels as the library does (C's round, halves away from zero), so that
what it hands over has the library's size for odd images."""
import ctypes as C
import ctypes.util

import numpy as np
import pytest

import dpe_b200 as D
import edges as E
import helpers as h
import oracle_py as O

SIZES = [(101, 77), (102, 78), (103, 75), (105, 82), (106, 87)]


def test_level_size_is_c_round():
    libm = C.CDLL(ctypes.util.find_library("m"))
    libm.roundf.restype, libm.roundf.argtypes = C.c_float, [C.c_float]
    for s in range(9):
        for n in list(range(1, 300)) + [801, 1601, 2050, 32767]:
            assert D.level_size(n, 1 << s) == int(libm.roundf(C.c_float(np.float32(n) * np.float32(1.0 / (1 << s)))))


@pytest.mark.parametrize("w,hgt", SIZES)
@pytest.mark.parametrize("scale", [1, 2])
def test_host_maps_have_the_level_size(w, hgt, scale):
    pytest.importorskip("cv2")
    rng = np.random.default_rng(w)
    g = np.full((hgt, w), 100, np.uint8)
    g[hgt // 4: hgt // 2, w // 4: w // 2] = 180
    g[rng.random((hgt, w)) < 0.02] = 30
    edge, label = E.level_inputs(g, 1 << scale)
    want = O.edge_labels(g, scale)
    assert label.shape == edge.shape == want.shape == (D.level_size(hgt, 1 << scale), D.level_size(w, 1 << scale))
    assert np.array_equal(label, want)
