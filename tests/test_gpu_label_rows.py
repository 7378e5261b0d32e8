"""Label maps (dpe_edge_labels) whose rows just fill, just pass and fall short of one step of Connect's
scan, for each of its block sizes, against the CPU restatement."""
import numpy as np
import pytest

import oracle_py as O
from test_gpu_label_sizes import _blobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [12, 31, 127, 128, 129, 132, 256, 511, 512, 513, 516, 1024, 2047, 2048, 2049])
@pytest.mark.parametrize("high_res", [False, True])
def test_row_widths(ctx, w, high_res):
    g = _blobs(w, 48, w)
    got, want = ctx.edge_labels(g, 0, high_res), O.edge_labels(g, 0, high_res)
    assert got.shape == want.shape and np.array_equal(got, want), int((got != want).sum())
