"""Rays inside a scattering medium search no further than the distance at which they
scatter. The lane-refill kernel of the binary layout searches without that bound and
decides afterwards, so its images are the yardstick: every other kernel's are equal, for
media from almost clear to opaque and for distances that are zero, infinite or NaN."""
import numpy as np
import pytest

from illume_gb300 import _capi as C
from illume_gb300 import synth
from illume_gb300.api import Context, HostScene, Renderer
from illume_gb300.scenedata import Material, Mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scattering,absorption", [(0.0, 0.1), (-1.0, 0.1), (1e-6, 0.01), (0.02, 0.01), (1.0, 0.05), (1e3, 0.0),
                                                   (1e30, 0.0)])
@pytest.mark.parametrize("isect", [C.ISECT_MT, C.ISECT_WATERTIGHT])
def test_bounded_search_gives_the_unbounded_image(scattering, absorption, isect):
    s = synth.cornell_scene(96, 72, spheres=False)
    P, T = synth.displaced_icosphere(12, 3)
    med = s.add_medium(np.full(3, absorption), scattering, 0.5)
    glass = s.add_material(Material(C.MAT_REFRACTIVE, s.constant((1, 1, 1)), s.constant((1e-4,) * 3), ior=1.3, medium=med))
    M = np.zeros((3, 4), np.float32)
    M[:, :3], M[:, 3] = np.eye(3) * 120.0, (277.5, 140.0, 277.5)
    s.add_instance(s.add_mesh(Mesh(P, T)), glass, M)
    s.add_sphere((420.0, 90.0, 130.0), 80.0, glass)
    ctx = Context(0)
    scene = HostScene.from_data(ctx, s)

    def image(**kw):
        r = Renderer(ctx, scene, spp=4, max_depth=24, width=96, height=72, intersector=isect, accum_mode=C.ACCUM_FP64, **kw)
        out = r.render(sums=True)
        r.close()
        return out["sum"], out["stats"].rays

    ref, rays = image(bvh_kind=C.BVH_BINARY, trace_variant=4)
    for kw in (dict(bvh_kind=C.BVH_WIDE4), dict(bvh_kind=C.BVH_WIDE4, trace_variant=4), dict(bvh_kind=C.BVH_BINARY),
               dict(bvh_kind=C.BVH_WIDE8), dict(bvh_kind=C.BVH_WIDE4, queue_slots=4096)):
        got, n = image(**kw)
        assert np.array_equal(ref, got, equal_nan=True) and n == rays
    ctx.close()
