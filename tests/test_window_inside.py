"""CPU test of window_inside (dpe_device.cuh), which decides that a strong window's taps need no clamp: no
tap of a window that it clears may leave the padded image, also where the projective depth nearly vanishes
at a corner of the window.  The arithmetic is the tap loop's, compiled for the host."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "kernel_host", "window_host.cpp")
W, H = 640, 480


@pytest.fixture(scope="module")
def host_lib(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("window") / "libwindow_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-fPIC", "-shared",
                    "-I/usr/local/cuda/include", SRC, "-o", lib], check=True)
    return C.CDLL(lib)


def _windows(n, near, rng):
    """Random windows whose smallest depth over the taps is about `near` times the centre's, and whose
    numerators come close to what window_inside lets pass (or lie well within)."""
    f = np.float32
    w = np.zeros((n, 11), f)
    w[:, 0] = rng.integers(0, W, n)
    w[:, 1] = rng.integers(0, H, n)
    w[:, 2:4] = rng.random((n, 2))
    zc = 10.0 ** rng.uniform(-2, 2, n) * rng.choice([-1, 1], n)
    share = rng.random(n)
    s = np.abs(zc) * (1 - near * rng.uniform(0.5, 2, n)) / 5.0
    w[:, 8], w[:, 9], w[:, 10] = zc, s * share * rng.choice([-1, 1], n), s * (1 - share) * rng.choice([-1, 1], n)
    den = np.abs(zc) - 5 * (np.abs(w[:, 9].astype(np.float64)) + np.abs(w[:, 10].astype(np.float64)))
    for k, (c, size) in enumerate(((0, W), (1, H))):
        room = np.minimum(w[:, c], size - 2 - w[:, c]).astype(np.float64)
        total = np.maximum(den, 0) * np.maximum(room, 0) / 5.0 * rng.uniform(0.5, 1.0, n)
        part = rng.random(n)
        w[:, 4 + k] = total * part * rng.choice([-1, 1], n)
        w[:, 6 + k] = total * (1 - part) * rng.choice([-1, 1], n)
    return w


@pytest.mark.parametrize("near", [0.9, 0.3, 1e-1, 1e-2, 3e-3, 1e-3, 1e-4, 1e-5, 1e-6, 1e-7])
def test_cleared_windows_stay_in_the_padded_image(host_lib, near):
    rng = np.random.default_rng(int(1 / near))
    w = _windows(20000, near, rng)
    inside = np.zeros(len(w), np.int32)
    span = np.zeros((len(w), 4), np.int32)
    host_lib.host_window_inside(W, H, len(w), w.ctypes.data_as(C.c_void_p), inside.ctypes.data_as(C.c_void_p),
                                span.ctypes.data_as(C.c_void_p))
    ok = (span[:, 0] >= 0) & (span[:, 1] <= W + 1) & (span[:, 2] >= 0) & (span[:, 3] <= H + 1)
    bad = (inside == 1) & ~ok
    print(f"smallest depth {near:g} of the centre's: {inside.mean():.3f} cleared, {int(bad.sum())} of them leave")
    assert not bad.any()
    if near >= 1e-2:
        assert inside.mean() > 0.3  # ordinary windows are cleared
