"""CPU test: strong windows whose deformable centre window has more taps than the strong window itself
(use_radius takes a step of max(2, 2 r / 5): radius 6 and 7 give 7 x 7 and 8 x 8 taps).  The kernels' source on
the host gives the oracle's bits for them."""
import numpy as np
import pytest

import dpe_b200 as D
import helpers as h
import oracle_py as O
from test_kernel_host import _assert_identical, _run, host_lib  # noqa: F401  (fixture)


def wide_center_call(radius, step, weak_radius):
    ws = h.S.make_scene("small_weak", seed=2)
    ref = 1
    images, cams, srcs = h.view_inputs(ws, ref)
    edge, low, label = h.synthetic_edges(ws.gray[ref])
    rng = np.random.default_rng(4)
    hgt, w = images[0].shape
    state = np.ascontiguousarray(np.concatenate([ws.normal[ref], ws.depth[ref][..., None]], -1).astype(np.float32))
    weak = rng.choice(3, (hgt, w), p=[0.2, 0.75, 0.05]).astype(np.uint8)
    p = h.refine_params(ws, len(images), level=1, state=D.REFINE_INIT, geom=False)
    p.max_iterations = 1
    p.strong_radius, p.strong_increment, p.weak_radius = radius, step, weak_radius
    kw = dict(plane_in=state, views_in=np.full((hgt, w), (1 << len(srcs)) - 1, np.uint32), weak_in=weak, edge=edge,
              edge_low=low, label=label, seed=7)
    return images, cams, p, kw


CASES = [(5, 2, 5), (6, 3, 5), (7, 3, 5), (9, 4, 5), (12, 5, 5), (7, 3, 0)]


@pytest.mark.parametrize("radius,step,weak_radius", CASES)
def test_wide_center(host_lib, radius, step, weak_radius):  # noqa: F811
    images, cams, p, kw = wide_center_call(radius, step, weak_radius)
    _assert_identical(_run(host_lib, images, cams, p, **kw), O.pm_run(images, cams, p, **kw))
