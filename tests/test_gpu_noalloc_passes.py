"""The allocation-free entry point renders several samples per pass where its fixed array
and the path kernel's range allow it. The sums equal a renderer's FP32 sums bit for bit:
one sample, a last pass that is smaller, the largest image, a depth of 0, a later first
sample, and the layouts that run one sample per pass."""
import ctypes

import numpy as np
import pytest

from illume_gb300 import _capi as C
from illume_gb300 import synth
from illume_gb300.api import Context, HostScene, Renderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp,depth,begin,kind", [
    (1, 1, 1, 5, 0, C.BVH_WIDE4), (33, 17, 40, 6, 0, C.BVH_WIDE4), (256, 256, 7, 4, 0, C.BVH_WIDE4),
    (200, 150, 9, 10, 3, C.BVH_WIDE4), (64, 40, 2, 0, 0, C.BVH_WIDE4), (64, 40, 0, 4, 0, C.BVH_WIDE4),
    (120, 90, 3, 5, 1, C.BVH_BINARY)])
def test_sums_equal_a_renderers(w, h, spp, depth, begin, kind):
    import torch

    ctx = Context(0)
    scene = HostScene.from_data(ctx, synth.traversal_scene(tris=2_000, env_size=(64, 32)))
    p = scene.default_params(spp, depth)
    p.width, p.height, p.sample_begin, p.bvh_kind, p.seed = w, h, begin, kind, 9
    sums = torch.full((w * h, 3), 5.0, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):   # the array keeps the first call's contents
        C.check(C.lib().illume_render_noalloc(ctx.handle, scene.handle, ctypes.byref(p), sums.data_ptr()))
    torch.cuda.synchronize()
    if spp == 0:
        assert (sums == 0).all()
    else:
        r = Renderer(ctx, scene, params=p)
        assert np.array_equal(sums.cpu().numpy(), r.render(sums=True)["sum"].astype(np.float32), equal_nan=True)
        r.close()
    ctx.close()
