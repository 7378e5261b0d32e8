"""Label maps (dpe_edge_labels) on both sides of the threshold from which a Hough round takes several
points' votes (a shorter side of 60 pixels of the halved map), with one block, a cluster and global counts,
against the CPU restatement."""
import numpy as np
import pytest

import oracle_py as O
from test_gpu_label_sizes import _blobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,hgt", [(200, 58), (200, 62), (200, 118), (200, 120), (200, 122), (900, 118), (900, 122),
                                   (1600, 110), (1600, 124), (6000, 100), (6000, 126)])
def test_votes_of_a_round(ctx, w, hgt):
    g = _blobs(w, hgt, w + hgt)
    got, want = ctx.edge_labels(g, 0, False), O.edge_labels(g, 0, False)
    assert got.shape == want.shape and np.array_equal(got, want), int((got != want).sum())
