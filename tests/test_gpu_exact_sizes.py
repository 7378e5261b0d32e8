"""The exact build against the CPU oracle where the per-view kernels' layouts have edges: images that
fill no block, one and many sources (cost rows beyond the shared memory that needs no opt-in), every
image storage, window sizes other than the 6 x 6 one that has its own loop.  Identical bits."""
import numpy as np
import pytest

import dpe_b200 as D
import helpers as h
import oracle_py as O
from test_gpu_exact import _same, xctx  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


def _scene(w, hgt, views, seed):
    f = 0.82 * w
    return h.S.make_scene(h.S.SceneSpec(width=w, height=hgt, n_views=views, fx=f, fy=f, cx=w / 2.0, cy=hgt / 2.0,
                                        tex_freq=0.04 * w, step_deg=min(10.0, 90.0 / views)), seed=seed)


def _images(scene, level):
    imgs = [np.ascontiguousarray(g.astype(np.float32)) for g in scene.gray]
    if level:  # values that are no 16-bit floats: the FP32 storage
        imgs = [np.ascontiguousarray((i + np.roll(i, 1, 1)) * np.float32(1.0 / 3.0)) for i in imgs]
    return imgs


@pytest.mark.parametrize("w,hgt,views,level,radius", [
    (16, 16, 2, False, 5), (33, 17, 3, True, 5), (47, 50, 32, False, 5), (64, 48, 12, True, 5),
    (40, 31, 4, False, 4), (35, 40, 4, True, 3)])
def test_first_init_sizes(xctx, w, hgt, views, level, radius):  # noqa: F811
    sc = _scene(w, hgt, views, seed=w)
    images, cams = _images(sc, level), [h.S.camera_struct(sc, i) for i in range(views)]
    p = h.first_init_params(sc, views)
    p.strong_radius = radius
    _same(xctx.pm_run(images, cams, p, seed=9), O.pm_run(images, cams, p, seed=9), f"{w}x{hgt}x{views}")


@pytest.mark.parametrize("w,hgt,views,level,geom", [(33, 29, 2, False, False), (61, 40, 18, True, True),
                                                    (96, 64, 5, False, True)])
def test_refine_sizes(xctx, w, hgt, views, level, geom):  # noqa: F811
    sc = _scene(w, hgt, views, seed=w + 1)
    images, cams = _images(sc, level), [h.S.camera_struct(sc, i) for i in range(views)]
    rng = np.random.default_rng(w)
    state = np.concatenate([sc.normal[0], sc.depth[0][..., None]], -1).astype(np.float32)
    state[..., 3] *= (1 + 0.02 * rng.standard_normal((hgt, w))).astype(np.float32)
    state[4:8, 4:20] = state[4, 4]  # equal planes side by side: candidates that share a cost row
    weak = rng.choice(3, (hgt, w), p=[0.3, 0.6, 0.1]).astype(np.uint8)
    edge, low, label = h.synthetic_edges(sc.gray[0])
    p = h.refine_params(sc, views, level=2, state=D.REFINE_ITER if geom else D.REFINE_INIT, geom=geom)
    kw = dict(plane_in=state, views_in=rng.integers(0, 2 ** (views - 1), (hgt, w)).astype(np.uint32), weak_in=weak,
              edge=edge, edge_low=low, label=label, seed=78)
    if geom:
        kw["depths"] = [np.ascontiguousarray(sc.depth[i].astype(np.float32)) for i in range(views)]
    _same(xctx.pm_run(images, cams, p, **kw), O.pm_run(images, cams, p, **kw), f"refine {w}x{hgt}x{views}")


@pytest.mark.parametrize("rotate,high_res,label,limit,weak_share", [(1, 1, 1, 1, 0.9), (2, 0, 1, 1, 0.5),
                                                                    (3, 1, 0, 1, 0.2), (4, 0, 0, 0, 0.6)])
def test_neighbour_search_options(xctx, rotate, high_res, label, limit, weak_share):  # noqa: F811
    """GenNeighbours and the plane fit: few and many rays, short and long line walks, with and without
    labels, edge limits and (where almost everything is WEAK) enough strong points."""
    w, hgt, views = 90, 70, 4
    sc = _scene(w, hgt, views, seed=rotate)
    images, cams = _images(sc, True), [h.S.camera_struct(sc, i) for i in range(views)]
    rng = np.random.default_rng(rotate)
    state = np.concatenate([sc.normal[0], sc.depth[0][..., None]], -1).astype(np.float32)
    weak = rng.choice(2, (hgt, w), p=[weak_share, 1 - weak_share]).astype(np.uint8)
    edge, low, lab = h.synthetic_edges(sc.gray[0], 0.04)
    lab = np.where(lab == 0, 0, 1 + (np.arange(w)[None, :] > w // 2)).astype(np.int32)
    p = h.refine_params(sc, views, level=2, state=D.REFINE_ITER, geom=True)
    p.rotate_time, p.high_res_img, p.use_label, p.use_limit = rotate, high_res, label, limit
    kw = dict(plane_in=state, views_in=rng.integers(1, 2 ** (views - 1), (hgt, w)).astype(np.uint32), weak_in=weak,
              edge=edge, edge_low=low, label=np.ascontiguousarray(lab),
              depths=[np.ascontiguousarray(sc.depth[i].astype(np.float32)) for i in range(views)], seed=5)
    _same(xctx.pm_run(images, cams, p, **kw), O.pm_run(images, cams, p, **kw), f"rotate {rotate}")
