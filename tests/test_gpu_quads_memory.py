"""A call whose 16-bit footprints do not fit into the device memory that is left samples the FP32 images
instead, with the same results; with FP16 or BF16 staging asked for it runs out of memory."""
import numpy as np
import pytest

import dpe_b200 as D
import helpers as h
from test_gpu_exact_sizes import _images, _scene

pytestmark = pytest.mark.gpu

W, H, N = 960, 720, 17


def test_footprints_that_do_not_fit():
    import torch

    sc = _scene(W, H, N, seed=1)
    cams = [h.S.camera_struct(sc, i) for i in range(N)]
    images = [torch.from_numpy(np.ascontiguousarray(g)).cuda() for g in _images(sc, 0)]
    p = h.first_init_params(sc, N, iters=1)

    out = dict(plane=torch.empty((H, W, 4), device="cuda"), weak=torch.empty((H, W), dtype=torch.uint8, device="cuda"),
               views=torch.empty((H, W), dtype=torch.int32, device="cuda"), costs=torch.empty((H, W), device="cuda"))

    def run(ctx):
        for o in out.values():
            o.zero_()
        torch.cuda.synchronize()
        ctx.pm_run(images, cams, p, seed=5, memory=D.MEM_DEVICE, out=dict(out))
        return [o.cpu().numpy() for o in out.values()]

    load = D.Context(0)  # every kernel of the call is loaded, in each storage
    for i in images:
        i.div_(3.0)
    torch.cuda.synchronize()
    run(load)
    for i in images:
        i.mul_(3.0).round_()
    torch.cuda.synchronize()
    want = run(load)
    load.close()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    ctx = D.Context(0)
    run(ctx)
    torch.cuda.empty_cache()
    need = free - torch.cuda.mem_get_info()[0]
    ctx.close()
    quads = 8 * (N - 1) * (W + 2) * (H + 2)
    assert need > quads
    keep = torch.empty(torch.cuda.mem_get_info()[0] - (need - quads // 2), dtype=torch.uint8, device="cuda")
    ctx = D.Context(0)
    try:
        got = run(ctx)
        assert all(np.array_equal(g, w, equal_nan=True) for g, w in zip(got, want))
        ctx.set_options(staging=D.STAGE_BF16)
        with pytest.raises(D.DPEError) as e:
            run(ctx)
        assert e.value.status == D.ERR_OUT_OF_MEMORY
    finally:
        ctx.close()
        del keep
        torch.cuda.empty_cache()
