"""The default 4-wide trace and occlusion kernels of the wavefront stages, which passes of at
most 2^18 paths never launch (the path kernel takes them): each triangle test's instance
and the watertight one for overlapping tables, on scenes on both sides of the sorted
instance walk, against the binary layout's images. A path-regenerating pass runs every
bounce through them at any size; a pass above 2^18 paths its first two at least. The
launch counts show the route."""
import numpy as np
import pytest

from illume_gb300 import _capi as C
from illume_gb300.api import HostScene, Renderer
from test_gpu_trace_kernels import scene_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("instances", [0, 1, 2, 3, 16, 17])
@pytest.mark.parametrize("estimator", [C.ESTIMATOR_REFERENCE, C.ESTIMATOR_NEE])
@pytest.mark.parametrize("isect", [C.ISECT_MT, C.ISECT_WATERTIGHT])
def test_images_equal_the_binary_layouts(ctx, instances, estimator, isect):
    scene = HostScene.from_data(ctx, scene_of(instances))
    depth, stages = 9, 3 if estimator == C.ESTIMATOR_NEE else 2

    def image(kind, w, h, spp, **kw):
        r = Renderer(ctx, scene, spp=spp, max_depth=depth, width=w, height=h, intersector=isect, estimator=estimator,
                     accum_mode=C.ACCUM_FP64, bvh_kind=kind, **kw)
        out = r.render(sums=True)
        r.close()
        return out["sum"], out["stats"]

    # 37 x 29: 33 warps and a part of one per sample; queues of 701 rays
    want, ws = image(C.BVH_BINARY, 37, 29, 6)
    for engines in (1, 2):
        got, gs = image(C.BVH_WIDE4, 37, 29, 6, queue_slots=701, engines=engines)
        assert gs.rays == ws.rays and np.array_equal(got, want, equal_nan=True)
        # regeneration: 5 launches a pass and stages + 2 an iteration, of which 6,438 paths in
        # batches of at most 701 take 10
        assert gs.kernel_launches >= engines * 5 + (stages + 2) * 10
    # 521 x 509: 2^18 + 3,045 paths a sample
    want, ws = image(C.BVH_BINARY, 521, 509, 4)
    for engines, per_pass, passes in ((1, 1, 4), (2, 2, 4)):
        got, gs = image(C.BVH_WIDE4, 521, 509, 4, engines=engines, samples_per_pass=per_pass)
        assert gs.rays == ws.rays and np.array_equal(got, want, equal_nan=True)
        # plan, camera rays, accumulation, advance, the stages, hand-over at bounces 2, 4 and 8
        assert gs.kernel_launches == passes * (4 + stages * depth + 3)
    scene.close()
