"""The storages that a call's source images can take.  Texels that FP16 does not hold: FP16 staging against FP32
staging is then a comparison of two storages (levels of exact halves and quarters take FP16 texels by
themselves).  Quarters, which FP16 holds and BF16 does not, and batches whose problems take different
storages, against the CPU oracle (exact build: identical bits)."""
import numpy as np
import pytest

import dpe_b200 as D
import helpers as h
import oracle_py as O
from test_gpu_exact import _same, xctx  # noqa: F401  (fixture)
from test_gpu_exact_sizes import _scene

pytestmark = pytest.mark.gpu


def _texels(sc, kind):
    imgs = [np.ascontiguousarray(g.astype(np.float32)) for g in sc.gray]
    if kind == "quarters":  # a halved level: averages of four 8-bit values
        imgs = [(i + np.roll(i, 1, 1) + np.roll(i, 1, 0) + np.roll(i, (1, 1), (0, 1))) * np.float32(0.25) for i in imgs]
    elif kind == "thirds":
        imgs = [(i + np.roll(i, 1, 1)) * np.float32(1.0 / 3.0) for i in imgs]
    return [np.ascontiguousarray(i) for i in imgs]


def _exact(imgs):
    """Whether FP16, and whether BF16, hold every source texel."""
    f16 = all(np.array_equal(i.astype(np.float16).astype(np.float32), i) for i in imgs[1:])
    return f16, all(not (i.view(np.uint32) & 0xFFFF).any() for i in imgs[1:])


KINDS = {"whole": (True, True), "quarters": (True, False), "thirds": (False, False)}


def _call(kind, w, hgt, views, geom):
    sc = _scene(w, hgt, views, seed=w + views)
    images, cams = _texels(sc, kind), [h.S.camera_struct(sc, i) for i in range(views)]
    assert _exact(images) == KINDS[kind]
    if geom is None:
        return images, cams, h.first_init_params(sc, views), dict(seed=9)
    rng = np.random.default_rng(w)
    state = np.concatenate([sc.normal[0], sc.depth[0][..., None]], -1).astype(np.float32)
    state[..., 3] *= (1 + 0.02 * rng.standard_normal((hgt, w))).astype(np.float32)
    weak = rng.choice(3, (hgt, w), p=[0.3, 0.6, 0.1]).astype(np.uint8)
    edge, low, label = h.synthetic_edges(sc.gray[0])
    p = h.refine_params(sc, views, level=2, state=D.REFINE_ITER if geom else D.REFINE_INIT, geom=geom)
    kw = dict(plane_in=state, views_in=rng.integers(0, 2 ** (views - 1), (hgt, w)).astype(np.uint32), weak_in=weak,
              edge=edge, edge_low=low, label=label, seed=78)
    if geom:
        kw["depths"] = [np.ascontiguousarray(sc.depth[i].astype(np.float32)) for i in range(views)]
    return images, cams, p, kw


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("geom", [None, False, True])
def test_storage_matches_oracle(xctx, kind, geom):  # noqa: F811
    images, cams, p, kw = _call(kind, 61, 47, 4, geom)
    _same(xctx.pm_run(images, cams, p, **kw), O.pm_run(images, cams, p, **kw), f"{kind} {geom}")


@pytest.mark.parametrize("kinds", [("whole", "quarters"), ("quarters", "quarters"), ("quarters", "thirds", "whole")])
@pytest.mark.parametrize("geom", [None, True])
def test_batch_of_storages(xctx, kinds, geom):  # noqa: F811
    calls = [_call(k, 61 - 8 * i, 47 + 4 * i, 4, geom) for i, k in enumerate(kinds)]
    got = xctx.pm_run_batch([dict(images=i, cameras=c, params=p, **kw) for i, c, p, kw in calls])
    for k, r, (i, c, p, kw) in zip(kinds, got, calls):
        _same(r, O.pm_run(i, c, p, **kw), f"batch {kinds} {k} {geom}")


@pytest.mark.parametrize("staging", [D.STAGE_FP16, D.STAGE_BF16])
def test_rounded_texels(ctx, small_scene, staging):
    """16-bit staging of texels that neither format holds.  FP16 moves a texel below 256 by at most 1/16 of a grey
    level, far below what the images' noise does to a cost; the bars are those of test_gpu_forms.py's comparison:
    0.98 of the depths for FP16, the accuracy for both."""
    images, cams, _ = h.view_inputs(small_scene, 1)
    images = [np.ascontiguousarray((i + np.roll(i, 1, 1) + np.roll(i, 1, 0)) * np.float32(1.0 / 3.0)) for i in images]
    assert _exact(images) == (False, False)
    p = h.first_init_params(small_scene, len(images))
    want = ctx.pm_run(images, cams, p, seed=32)
    try:
        ctx.set_options(staging=staging)
        got = ctx.pm_run(images, cams, p, seed=32)
    finally:
        ctx.set_options()
    assert not np.array_equal(got["plane"], want["plane"])  # another storage was sampled
    agree = h.rel_depth_agreement(got["plane"][..., 3], want["plane"][..., 3], 1e-3)
    gt = small_scene.depth[1]
    acc = lambda o: float((np.abs(o["plane"][..., 3] - gt) / gt < 0.01).mean())
    print(f"staging {staging}: depth agreement with FP32 {agree:.4f}; within 1% of GT {acc(want):.4f} {acc(got):.4f}")
    if staging == D.STAGE_FP16:
        assert agree >= 0.98
    assert acc(got) >= acc(want) - 0.02
