"""The strong update's launches all take the driver's carveout: none of them is spent on trying others."""
import pytest

import dpe_b200 as D
import helpers as h

pytestmark = pytest.mark.gpu


def test_one_setting(small_scene):
    images, cams, _ = h.view_inputs(small_scene, 0)
    p = h.first_init_params(small_scene, len(images))
    c = D.Context(0)
    try:
        for _ in range(4):
            c.pm_run(images, cams, p, seed=1)
        e = next(e for e in c.tuning() if e["kernel"] == "k_strong_update")
    finally:
        c.close()
    assert (e["candidates"], e["chosen"], e["carveout"]) == (1, 0, -1)
