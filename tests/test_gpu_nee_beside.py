"""A bounce's occlusion rays run beside the next bounce's closest-hit rays. The regeneration
loop runs the same stages one after another; images and ray counts are equal bit for bit,
for depths with no, one and many bounces side by side, with hand-over to the path kernel and
without (the binary layout), on one engine and on several."""
import numpy as np
import pytest

from illume_gb300 import _capi as C
from illume_gb300 import synth
from illume_gb300.api import Context, HostScene, Renderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["ground", "cornell"])
@pytest.mark.parametrize("bvh", [C.BVH_WIDE4, C.BVH_BINARY])
def test_images_equal_the_sequential_stages(kind, bvh):
    ctx = Context(0)
    data = synth.traversal_scene(tris=2_000, env_size=(64, 32)) if kind == "ground" else synth.cornell_scene(64, 64)
    sc = HostScene.from_data(ctx, data)

    def image(queue, w, h, spp, depth, engines):
        r = Renderer(ctx, sc, spp=spp, max_depth=depth, width=w, height=h, estimator=1, bvh_kind=bvh,
                     accum_mode=C.ACCUM_FP64, engines=engines, queue_slots=queue)
        out = [r.render(sums=True) for _ in range(2)]
        r.close()
        assert np.array_equal(out[0]["sum"], out[1]["sum"], equal_nan=True)
        return out[0]["sum"], out[0]["stats"].rays

    for w, h, spp, depth, engines in ((33, 21, 3, 1, 1), (512, 513, 1, 2, 1), (300, 301, 5, 3, 1), (512, 512, 4, 9, 1),
                                      (640, 480, 6, 25, 2)):
        a, b = image(0, w, h, spp, depth, engines), image(w * h // 2, w, h, spp, depth, 1)
        assert a[1] == b[1]
        assert np.array_equal(a[0], b[0], equal_nan=True)
    ctx.close()
