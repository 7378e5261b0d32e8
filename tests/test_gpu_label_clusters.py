"""Label maps (dpe_edge_labels) for every number of blocks that share a region's Hough counts: 1, 2, 4 and 8, and
counts in global memory, against the CPU restatement.  The rule is restated here, so that a change of the limit
cannot drop a path from the sizes."""
import math

import numpy as np
import pytest

import oracle_py as O
from test_gpu_label_sizes import _blobs

pytestmark = pytest.mark.gpu

SHARED, ANGLES = 200 * 1024, 180


def _split(w, hgt, high_res):
    """Blocks per region for the halved map of a w x hgt image; 0: counts in global memory."""
    for _ in range(2 if high_res else 1):
        w, hgt = w // 2, hgt // 2
    bins = min(w + math.ceil(math.hypot(w, hgt)) + 2, (w + hgt) * 2 + 1 - (w + hgt - w))
    rest = 2 * (max(w, hgt) + 2) * 4 + (w * hgt + 31) // 32 * 4
    return next((k for k in (1, 2, 4, 8) if rest + -(-ANGLES // k) * bins * 2 <= SHARED), 0)


@pytest.mark.parametrize("w,hgt,high_res,split", [
    (400, 300, False, 1), (640, 480, False, 2), (1000, 700, False, 4), (1600, 1200, False, 8), (3200, 2400, True, 8),
    (2200, 1800, False, 0), (4800, 3600, True, 0)])
def test_counts_shared_by_blocks(ctx, w, hgt, high_res, split):
    assert _split(w, hgt, high_res) == split
    g = _blobs(w, hgt, w)
    got, want = ctx.edge_labels(g, 0, high_res), O.edge_labels(g, 0, high_res)
    assert got.shape == want.shape and np.array_equal(got, want), int((got != want).sum())
