"""Label maps (dpe_edge_labels) of images whose Hough counts take just under and just over the 48 KB of
shared memory that need no opt-in, the kernel's static part among them; against the CPU restatement."""
import numpy as np
import pytest

import oracle_py as O
from test_gpu_label_sizes import _blobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,hgt,high_res", [(w, int(0.75 * w), False) for w in range(106, 122, 2)] +
                         [(w, int(0.55 * w), True) for w in range(224, 256, 4)])
def test_counts_near_the_limit(ctx, w, hgt, high_res):
    g = _blobs(w, hgt, w)
    got, want = ctx.edge_labels(g, 0, high_res), O.edge_labels(g, 0, high_res)
    assert got.shape == want.shape and np.array_equal(got, want), int((got != want).sum())
