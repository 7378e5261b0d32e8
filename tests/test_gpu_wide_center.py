"""The GPU against the CPU oracle where the deformable centre window has more taps than the strong window
(exact build: identical bits)."""
import pytest

import oracle_py as O
from test_gpu_exact import _same, xctx  # noqa: F401  (fixture)
from test_wide_center import CASES, wide_center_call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius,step,weak_radius", CASES)
def test_wide_center(xctx, radius, step, weak_radius):  # noqa: F811
    images, cams, p, kw = wide_center_call(radius, step, weak_radius)
    _same(xctx.pm_run(images, cams, p, **kw), O.pm_run(images, cams, p, **kw), f"radius {radius} step {step}")
