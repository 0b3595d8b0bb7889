"""Which passes run as two halves (seen in the launch count): those of a room, five or six
walls that neither shine nor let light through, whatever stands in it; in open scenes, where
halves lose up to 15%, and under an environment a pass runs whole. The image is the same."""
import numpy as np
import pytest

from illume_gb300 import _capi as C
from illume_gb300 import synth
from illume_gb300.api import HostScene, Renderer
from illume_gb300.scenedata import Material, Mesh, SceneData, Texture

pytestmark = pytest.mark.gpu

FACES = [(0, 2, 6, 4), (1, 5, 7, 3), (0, 4, 5, 1), (2, 3, 7, 6), (4, 6, 7, 5), (0, 1, 3, 2)]


def scene(walls=0, wall=C.MAT_LAMBERT, size=1.0, far=False, env=False):
    s = SceneData()
    rng = np.random.default_rng(3)
    body = s.add_mesh(Mesh(*synth.displaced_icosphere(16, 5)))   # 5,120 triangles
    s.add_instance(body, synth.mixed_material(s, rng))
    P, T, UV = synth.quad(1.0, 1.9)
    lamp = s.add_material(Material(C.MAT_EMISSIVE, s.constant((9, 9, 8)), s.constant((1e-4,) * 3)))
    s.add_instance(s.add_mesh(Mesh(P, T)), lamp)
    if far:
        s.add_sphere((40.0, 0.0, 0.0), 1.0, lamp)
    m = s.add_material(Material(wall, s.constant((0.7,) * 3), s.constant((1e-4,) * 3), ior=1.5))
    c = np.array([[2.0 if (i >> k) & 1 else -2.0 for k in range(3)] for i in range(8)], np.float32)
    for f in FACES[:walls]:
        q = c[list(f)]
        s.add_instance(s.add_mesh(Mesh((q.mean(0) + (q - q.mean(0)) * np.float32(size)).astype(np.float32),
                                       np.array([(0, 1, 2), (0, 2, 3)], np.int32))), m)
    if env:
        s.env_tex = s.add_texture(Texture(C.TEX_BITMAP, texels=synth.environment_map(1, 64, 32), hdr=1))
    s.camera_transform = synth.lookat((0.0, 0.3, -1.9), (0.0, 0.0, 0.0))
    s.ray_bias = 1e-4
    return s


@pytest.mark.parametrize("halves,kw", [
    (True, dict(walls=5)), (True, dict(walls=6)), (True, dict(walls=5, size=0.96)), (True, dict(walls=5, wall=C.MAT_PLASTIC)),
    (False, dict()), (False, dict(walls=4)), (False, dict(walls=5, size=0.9)), (False, dict(walls=6, wall=C.MAT_EMISSIVE)),
    (False, dict(walls=6, wall=C.MAT_REFRACTIVE)), (False, dict(walls=6, far=True)), (False, dict(walls=6, env=True))])
def test_rooms_run_as_halves(ctx, halves, kw):
    sc = HostScene.from_data(ctx, scene(**kw))
    out = []
    for engines in (0, 1):
        r = Renderer(ctx, sc, spp=1, max_depth=4, width=1024, height=1024, accum_mode=C.ACCUM_FP64, engines=engines)
        out.append(r.render(sums=True))
        r.close()
    a, b = out
    assert (a["stats"].kernel_launches > b["stats"].kernel_launches) == halves
    assert a["stats"].rays == b["stats"].rays and np.array_equal(a["sum"], b["sum"], equal_nan=True)
