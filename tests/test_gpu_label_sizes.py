"""Label maps (dpe_edge_labels) at the sizes where the device's layouts change, against the CPU
restatement: rows that fill less and more than one step of Connect's scan (2048 pixels), and Hough
counts that fit one block's shared memory, that 2, 4 or 8 blocks split, and that stay in global memory."""
import numpy as np
import pytest

import oracle_py as O

pytestmark = pytest.mark.gpu


def _blobs(w, hgt, seed):
    """Flat regions with straight and ragged borders: every kind of run, join and segment."""
    rng = np.random.default_rng(seed)
    img = np.full((hgt, w), 100, np.uint8)
    for _ in range(40):
        x, y = rng.integers(0, w), rng.integers(0, hgt)
        dx, dy = rng.integers(8, max(9, w // 3)), rng.integers(8, max(9, hgt // 2))
        img[y:y + dy, x:x + dx] = rng.integers(60, 200)
    noisy = rng.random((hgt, w)) < 0.02
    img[noisy] = rng.integers(0, 255, int(noisy.sum()))
    return img


@pytest.mark.parametrize("w,hgt,scale", [(64, 48, 0), (131, 97, 0), (2050, 60, 0), (4110, 40, 0), (800, 600, 1),
                                         (1600, 1200, 0), (3000, 1000, 2), (6000, 1600, 3), (9200, 128, 3)])
def test_label_sizes(ctx, w, hgt, scale):
    g = _blobs(w, hgt, w + scale)
    got, want = ctx.edge_labels(g, scale), O.edge_labels(g, scale)
    assert got.shape == want.shape and np.array_equal(got, want), int((got != want).sum())
