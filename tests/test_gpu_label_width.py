"""Label maps (dpe_edge_labels) of the widest images that they take: a halved map up to 14445 pixels on its
longer side, against the CPU restatement; wider ones are refused with an error."""
import numpy as np
import pytest

import dpe_b200 as D
import oracle_py as O
from test_gpu_label_sizes import _blobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,hgt,high_res", [(28890, 32, False), (28600, 120, False), (57700, 64, True)])
def test_widest_maps(ctx, w, hgt, high_res):
    g = _blobs(w, hgt, w)
    got, want = ctx.edge_labels(g, 0, high_res), O.edge_labels(g, 0, high_res)
    assert got.shape == want.shape and np.array_equal(got, want), int((got != want).sum())


def test_wider_maps_are_refused(ctx):
    with pytest.raises(D.DPEError) as e:
        ctx.edge_labels(_blobs(28900, 32, 1), 0, False)
    assert e.value.status == D.ERR_CUDA
    g = _blobs(640, 480, 2)
    assert np.array_equal(ctx.edge_labels(g, 0), O.edge_labels(g, 0))  # the context goes on
