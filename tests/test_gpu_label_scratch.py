"""Device memory that the label maps keep for an image with many large regions: the points of a region's
border are its own border's, not the map's."""
import numpy as np
import pytest

import dpe_b200 as D
import oracle_py as O

pytestmark = pytest.mark.gpu


def _checks(w, hgt, step):
    """Squares of two shades: every square is a region of its own."""
    y, x = np.mgrid[0:hgt, 0:w]
    return np.where((x // step + y // step) & 1, 180, 100).astype(np.uint8)


@pytest.mark.parametrize("w,hgt,scale,high_res,step", [(1600, 1200, 3, False, 32), (3200, 2400, 3, True, 80)])
def test_scratch_of_many_regions(w, hgt, scale, high_res, step):
    import torch

    g = _checks(w, hgt, step)
    ctx = D.Context(0)
    try:
        ctx.edge_labels(g[:64, :64].copy(), 0, high_res)  # the library's kernels are loaded
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        got = ctx.edge_labels(g, scale, high_res)
        used = free - torch.cuda.mem_get_info()[0]
    finally:
        ctx.close()
    want = O.edge_labels(g, scale, high_res)
    assert np.array_equal(got, want)
    n2 = (w // (4 if high_res else 2)) * (hgt // (4 if high_res else 2))
    regions = (w // step) * (hgt // step)
    print(f"{w}x{hgt}: {regions} squares, {used / 2**20:.0f} MiB")
    # per pixel of the halved map: at most 4 border points of 8 bytes for each of 8 blocks, and the rest of
    # the maps; per pixel of the image: input, halved copy, output; per region: its lines; the allocator's
    # own 2 MiB steps for two dozen buffers
    assert used <= n2 * (4 * 8 * 8 + 120) + w * hgt * 4 + regions * n2 + (64 << 20)
