"""Label maps (dpe_edge_labels) of images with odd sizes at coarser levels, in host and in device memory, against the
CPU restatement: the map is the library's size, which rounds halves up."""
import numpy as np
import pytest

import dpe_b200 as D
import oracle_py as O
from test_gpu_label_sizes import _blobs
from test_level_size import SIZES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,hgt", SIZES + [(801, 601), (803, 603)])
@pytest.mark.parametrize("scale", [1, 2, 3])
def test_odd_sizes(ctx, w, hgt, scale):
    import torch

    g = _blobs(w, hgt, w)
    want = O.edge_labels(g, scale)
    got = ctx.edge_labels(g, scale)
    assert got.shape == want.shape and np.array_equal(got, want)
    dev = torch.from_numpy(g).cuda()
    torch.cuda.synchronize()
    assert np.array_equal(ctx.edge_labels(dev, scale, memory=D.MEM_DEVICE).cpu().numpy(), want)
