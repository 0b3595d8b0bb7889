"""The default 4-wide trace and occlusion kernels exist once per triangle test (the
Moller-Trumbore one specialised for it). Their images equal those of the binary layout's
kernels, which read the test from their settings, for scenes on both sides of the sorted
instance walk (3 to 16 instances) and frames that leave partial warps."""
import numpy as np
import pytest

from illume_gb300 import _capi as C
from illume_gb300 import synth
from illume_gb300.api import Context, HostScene, Renderer
from illume_gb300.scenedata import Material, Mesh, SceneData, Texture

pytestmark = pytest.mark.gpu


def scene_of(instances):
    rng = np.random.default_rng(instances)
    s = SceneData()
    meshes = [s.add_mesh(Mesh(*synth.displaced_icosphere(f, 7 + f))) for f in (1, 6)]
    lamp = s.add_material(Material(C.MAT_EMISSIVE, s.constant((4, 4, 3)), s.constant((1e-4,) * 3)))
    for i in range(instances):
        M = np.zeros((3, 4))
        M[:, :3], M[:, 3] = synth.random_rotation(rng) * rng.uniform(0.5, 1.5), rng.uniform(-3, 3, 3)
        s.add_instance(meshes[i % 2], lamp if i == 1 else synth.mixed_material(s, rng), M.astype(np.float32))
    s.add_sphere((0.5, 2.0, 0.0), 0.7, s.add_material(Material(C.MAT_REFLECTIVE, s.constant((1, 1, 1)), s.constant((1e-4,) * 3))))
    s.env_tex = s.add_texture(Texture(C.TEX_BITMAP, texels=synth.environment_map(1, 64, 32), hdr=1))
    s.camera_transform = synth.lookat((0.0, 3.0, -9.0), (0.0, 0.0, 0.0))
    s.ray_bias = 1e-3
    return s


@pytest.mark.parametrize("instances", [0, 1, 2, 3, 16, 17])
@pytest.mark.parametrize("estimator", [C.ESTIMATOR_REFERENCE, C.ESTIMATOR_NEE])
@pytest.mark.parametrize("isect", [C.ISECT_MT, C.ISECT_WATERTIGHT])
def test_images_equal_the_binary_layouts(instances, estimator, isect):
    ctx = Context(0)
    scene = HostScene.from_data(ctx, scene_of(instances))

    def image(kind, w, h, spp):
        r = Renderer(ctx, scene, spp=spp, max_depth=9, width=w, height=h, intersector=isect, estimator=estimator,
                     accum_mode=C.ACCUM_FP64, bvh_kind=kind)
        out = r.render(sums=True)
        r.close()
        return out["sum"], out["stats"].rays

    for w, h, spp in ((1, 1, 1), (37, 29, 3)):
        a, na = image(C.BVH_WIDE4, w, h, spp)
        b, nb = image(C.BVH_BINARY, w, h, spp)
        assert na == nb and np.array_equal(a, b, equal_nan=True)
    ctx.close()


@pytest.mark.parametrize("instances", [1, 5, 17])
def test_overlapping_engines_give_one_engines_image(instances):
    # the watertight test has a kernel of its own where a pass's tables overlap
    ctx = Context(0)
    scene = HostScene.from_data(ctx, scene_of(instances))
    out = []
    for engines in (1, 2, 3):
        r = Renderer(ctx, scene, spp=7, max_depth=9, width=290, height=170, accum_mode=C.ACCUM_FP64, engines=engines)
        o = r.render(sums=True)
        out.append((o["sum"], o["stats"].rays))
        r.close()
    for s, n in out[1:]:
        assert n == out[0][1] and np.array_equal(s, out[0][0], equal_nan=True)
    ctx.close()
