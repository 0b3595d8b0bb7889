"""Shading reads face normals made at upload; a context with a budget makes none and
computes them at every hit. Both give the same image, for meshes with and without normals
and texture coordinates in one scene, degenerate triangles among them, and after the
geometry is uploaded again."""
import numpy as np
import pytest

from illume_gb300 import _capi as C
from illume_gb300 import synth
from illume_gb300.api import Context, HostScene, Renderer
from illume_gb300.scenedata import Material, Mesh, SceneData, Texture

pytestmark = pytest.mark.gpu


def world():
    s = SceneData()
    P, T = synth.displaced_icosphere(7, 4)
    T = np.concatenate([T, T[:2, [0, 0, 1]]]).astype(np.int32)          # no area, no normal
    N = (P / np.linalg.norm(P, axis=1, keepdims=True)).astype(np.float32)
    GP, GT, GUV = synth.quad(20.0, -1.2)
    tiny = s.constant((1e-4,) * 3)
    checker = s.add_texture(Texture(C.TEX_CHECKERBOARD, color=(0.8,) * 3, off=(0.2,) * 3, scale=(16.0, 16.0)))
    grey = s.add_material(Material(C.MAT_LAMBERT, s.constant((0.6,) * 3), tiny))
    gold = s.add_material(Material(C.MAT_ROUGHCONDUCTOR, s.constant((0,) * 3), s.constant((0.2,) * 3), eta=synth.GOLD_ETA,
                                   k=synth.GOLD_K, distribution=C.DIST_GGX))
    ground = s.add_material(Material(C.MAT_LAMBERT, checker, tiny))
    for k, (normals, mat) in enumerate(((None, gold), (N, grey), (None, grey))):
        M = np.eye(4)[:3].copy()
        M[0, 3] = 2.4 * (k - 1)
        s.add_instance(s.add_mesh(Mesh(P * np.float32(1.0 - 0.1 * k), T, normals=normals)), mat, M.astype(np.float32))
    s.add_instance(s.add_mesh(Mesh(GP, GT, texcoords=GUV)), ground)
    s.env_tex = s.add_texture(Texture(C.TEX_BITMAP, texels=synth.environment_map(1, 64, 32), hdr=1))
    s.camera_transform = synth.lookat((0.0, 1.5, -7.0), (0.0, 0.0, 0.0))
    s.ray_bias = 1e-4
    return s


@pytest.mark.parametrize("estimator", [C.ESTIMATOR_REFERENCE, C.ESTIMATOR_NEE])
@pytest.mark.parametrize("kind", [C.BVH_WIDE4, C.BVH_BINARY])
def test_made_and_computed_normals_agree(estimator, kind):
    out = []
    for budget in (0, 4 << 30):
        ctx = Context(0, hbm_budget_bytes=budget)
        scene = HostScene.from_data(ctx, world())
        for again in (False, True):
            if again:
                C.check(C.lib().illume_scene_upload(scene.handle, None))
            r = Renderer(ctx, scene, spp=6, max_depth=8, width=101, height=67, accum_mode=C.ACCUM_FP64, bvh_kind=kind,
                         estimator=estimator)
            out.append(r.render(sums=True)["sum"])
            r.close()
        ctx.close()
    for o in out[1:]:
        assert np.array_equal(out[0], o, equal_nan=True)
