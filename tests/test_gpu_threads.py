"""One context per host thread: calls whose kernels take different amounts of dynamic shared memory
(above the 48 KB that need no opt-in) run side by side, and give what they give alone.  The opt-in belongs
to the kernel function, process-wide: one thread's must not take back another's."""
import threading

import numpy as np
import pytest

import dpe_b200 as D
import helpers as h
from test_gpu_exact_sizes import _images, _scene
from test_gpu_label_sizes import _blobs

pytestmark = pytest.mark.gpu


def _side_by_side(works, repeats):
    """Runs every work (a function of a context) on a thread of its own, `repeats` times; each result has
    to be the one the work gives alone."""
    failures = []
    start = threading.Barrier(len(works))

    def go(work, ctx, want):
        try:
            start.wait()
            for _ in range(repeats):
                got = work(ctx)
                if not all(np.array_equal(g, w, equal_nan=True) for g, w in zip(got, want)):
                    failures.append("results differ")
        except D.DPEError as e:
            failures.append(str(e))

    contexts = [D.Context(0) for _ in works]
    try:
        threads = [threading.Thread(target=go, args=(w, c, w(c))) for w, c in zip(works, contexts)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        for c in contexts:
            c.close()
    assert not failures, (len(failures), failures[0])


def _labels(w, hgt, plain=False):
    """plain: one rectangle, a short call, so that many meet."""
    g = _blobs(w, hgt, w)
    if plain:
        g = np.full((hgt, w), 100, np.uint8)
        g[hgt // 4: 3 * hgt // 4, w // 4: 3 * w // 4] = 180
    return lambda ctx: [ctx.edge_labels(g, 0)]


def _first_call(views):
    sc = _scene(48, 32, views, seed=views)
    images, cams = _images(sc, 0), [h.S.camera_struct(sc, i) for i in range(views)]
    p = h.first_init_params(sc, views, iters=12)

    def run(ctx):
        r = ctx.pm_run(images, cams, p, seed=views)
        return [r["plane"], r["weak"], r["views"], r["costs"]]

    return run


@pytest.mark.parametrize("sizes,repeats", [([(400, 300, True), (440, 330, True), (480, 360, True), (520, 390, True)], 800),
                                           ([(400, 300), (1600, 1200)], 20)])
def test_label_maps(sizes, repeats):
    _side_by_side([_labels(*s) for s in sizes], repeats)


@pytest.mark.parametrize("views,repeats", [((22, 24, 28, 32), 60)])
def test_many_sources(views, repeats):
    _side_by_side([_first_call(v) for v in views], repeats)
