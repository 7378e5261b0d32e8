"""CPU test: low-resolution edge maps with more than 32767 columns or rows.  The kernels' source on the host
gives the oracle's bits for them."""
import numpy as np
import pytest

import dpe_b200 as D
import helpers as h
import oracle_py as O
from test_kernel_host import _assert_identical, _run, host_lib  # noqa: F401  (fixture)


def low_edge_call(shape, seed=5):
    """A weak-texture call whose low-resolution edge map has the given shape (sparse edges)."""
    ws = h.S.make_scene("small_weak", seed=2)
    ref = 1
    images, cams, srcs = h.view_inputs(ws, ref)
    edge, _, label = h.synthetic_edges(ws.gray[ref], 0.02)
    rng = np.random.default_rng(seed)
    hgt, w = images[0].shape
    low = (rng.random(shape) < 0.002).astype(np.uint8) * 255
    state = np.ascontiguousarray(np.concatenate([ws.normal[ref], ws.depth[ref][..., None]], -1).astype(np.float32))
    weak = rng.choice(2, (hgt, w), p=[0.3, 0.7]).astype(np.uint8)
    p = h.refine_params(ws, len(images), level=1, state=D.REFINE_INIT, geom=False)
    p.max_iterations = 1
    p.use_edge = 0  # every WEAK pixel keeps its edge limit
    kw = dict(plane_in=state, views_in=np.full((hgt, w), (1 << len(srcs)) - 1, np.uint32), weak_in=weak, edge=edge,
              edge_low=low, label=label, seed=7)
    return images, cams, p, kw


@pytest.mark.parametrize("shape", [(36, 40000), (40000, 48)])
def test_many_columns_or_rows(host_lib, shape):  # noqa: F811
    images, cams, p, kw = low_edge_call(shape)
    _assert_identical(_run(host_lib, images, cams, p, **kw), O.pm_run(images, cams, p, **kw))
