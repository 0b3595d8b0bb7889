"""Outputs reach the caller through page-locked staging memory when small and directly when
large, and host-buffer queries use kept device memory up to a limit: the same values on
both sides of each limit, in any order of sizes, with one renderer after another on a
context, and under a budget (where nothing is kept)."""
import numpy as np
import pytest

from illume_gb300 import _capi as C
from illume_gb300 import synth
from illume_gb300.api import Context, HostScene, Renderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (64, 48), (66, 66), (67, 66), (300, 200)])   # 65,340 and 66,330 bytes of images
@pytest.mark.parametrize("accum", [C.ACCUM_FP32, C.ACCUM_KAHAN, C.ACCUM_FP64])
def test_one_call_equals_its_parts(w, h, accum):
    ctx = Context(0)
    scene = HostScene.from_data(ctx, synth.cornell_scene(w, h))
    r = Renderer(ctx, scene, spp=3, max_depth=5, width=w, height=h, accum_mode=accum)
    whole = r.render(mean=True, sums=True, rgb8=True)
    other = Renderer(ctx, scene, spp=1, max_depth=2, width=16, height=16)
    other.render(rgb8=True)
    st = r.render_device()
    parts = r.read(mean=True, sums=True, rgb8=True)
    for k in ("mean", "sum", "sumsq", "rgb8"):
        assert np.array_equal(whole[k], parts[k])
        only = r.read(**{"mean": k == "mean", "sums": k.startswith("sum"), "rgb8": k == "rgb8"})
        assert np.array_equal(only[k], whole[k])
    assert whole["stats"].rays == st.rays and whole["stats"].paths == st.paths == 3 * w * h
    more = r.render_device(accumulate=True)      # the next three samples, on top
    assert more.rays > 0 and more.rays != 2 * st.rays
    prof = C.Profile()
    C.check(C.lib().illume_renderer_profile(r.handle, 0, C.ctypes.byref(prof)))
    assert r.render_device().rays == st.rays     # totals read elsewhere do not leak into a call's count
    other.close()
    r.close()
    ctx.close()


@pytest.mark.parametrize("budget", [0, 1 << 30])
def test_queries_of_any_size_in_any_order(budget):
    ctx = Context(0, hbm_budget_bytes=budget)
    scene = HostScene.from_data(ctx, synth.traversal_scene(tris=500, env_size=(16, 8)))
    rng = np.random.default_rng(1)
    n = 1_100_000                                # 70 MB of rays and hits: past what is kept
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = rng.normal(size=(n, 3)) * 3
    rays[:, 4:7] = -rays[:, :3] + rng.uniform(-1, 1, (n, 3))
    ref = scene.trace_closest(rays)
    for m in (1, 8_192, 8_193, 100, 40_000, 1_048_576, 5, 1_048_577, 64):
        got = scene.trace_closest(rays[:m])
        for k in got:
            assert np.array_equal(got[k], ref[k][:m])
    ctx.close()
