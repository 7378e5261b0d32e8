"""CPU test: a geometric call with a negative geom_factor, where costs can be negative and LocalRefine's
bounds do not hold.  The kernels' source on the host gives the oracle's bits for it too."""
import numpy as np
import pytest

import dpe_b200 as D
import helpers as h
import oracle_py as O
from test_kernel_host import _assert_identical, _run, host_lib  # noqa: F401  (fixture)


@pytest.mark.parametrize("factor", [-0.2, -1.0, 0.0, float("nan")])
def test_geom_factor_without_bounds(host_lib, factor):  # noqa: F811
    ws = h.S.make_scene("small_weak", seed=2)
    ref = 2
    images, cams, srcs = h.view_inputs(ws, ref)
    edge, low, label = h.synthetic_edges(ws.gray[ref])
    rng = np.random.default_rng(5)
    hgt, w = images[0].shape
    depth = ws.depth[ref] * (1 + 0.02 * rng.standard_normal((hgt, w)))
    state = np.ascontiguousarray(np.concatenate([ws.normal[ref], depth[..., None]], -1).astype(np.float32))
    weak = rng.choice(3, (hgt, w), p=[0.2, 0.75, 0.05]).astype(np.uint8)
    p = h.refine_params(ws, len(images), level=1, state=D.REFINE_ITER, geom=True)
    p.max_iterations = 1
    p.geom_factor = factor
    kw = dict(plane_in=state, views_in=np.full((hgt, w), (1 << len(srcs)) - 1, np.uint32), weak_in=weak, edge=edge,
              edge_low=low, label=label, seed=7,
              depths=[np.ascontiguousarray(ws.depth[i].astype(np.float32)) for i in [ref] + list(srcs)])
    _assert_identical(_run(host_lib, images, cams, p, **kw), O.pm_run(images, cams, p, **kw))
