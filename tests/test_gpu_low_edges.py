"""The GPU against the CPU oracle with low-resolution edge maps of more than 32767 columns or rows, and of the
usual quarter size (exact build: identical bits)."""
import pytest

import oracle_py as O
from test_gpu_exact import _same, xctx  # noqa: F401  (fixture)
from test_low_edges import low_edge_call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(36, 40000), (40000, 48), (36, 48), (361, 480)])
def test_low_edge_maps(xctx, shape):  # noqa: F811
    images, cams, p, kw = low_edge_call(shape)
    _same(xctx.pm_run(images, cams, p, **kw), O.pm_run(images, cams, p, **kw), f"low {shape}")
