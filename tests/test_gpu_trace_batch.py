"""Batches of closest-hit queries: few rays are spread over the warps, many run 32 to a
warp. The binary layout's hits are the yardstick for the 4-wide kernels, at the sizes where
the spread changes, and a caller's hit buffer may start at any 4-byte boundary."""
import numpy as np
import pytest

from illume_gb300 import _capi as C
from illume_gb300 import synth
from illume_gb300.api import Context, HostScene
from illume_gb300.scenedata import Material, Mesh, SceneData

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world():
    s = SceneData()
    rng = np.random.default_rng(3)
    grey = s.add_material(Material(C.MAT_LAMBERT, s.constant((0.5,) * 3), s.constant((1e-4,) * 3)))
    m = s.add_mesh(Mesh(*synth.displaced_icosphere(9, 5)))
    for i in range(4):
        M = np.zeros((3, 4))
        M[:, :3], M[:, 3] = synth.random_rotation(rng), rng.uniform(-2, 2, 3)
        s.add_instance(m, grey, M.astype(np.float32))
    s.add_sphere((0.0, 2.5, 0.0), 0.8, grey)
    ctx = Context(0)
    scene = HostScene.from_data(ctx, s)
    n = 194_600
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = rng.normal(size=(n, 3)) * 5
    rays[:, 4:7] = rng.uniform(-2, 2, (n, 3)) - rays[:, :3]
    rays[:, 4:7] /= np.linalg.norm(rays[:, 4:7], axis=1, keepdims=True)
    yield ctx, scene, rays
    ctx.close()


@pytest.mark.parametrize("isect", [C.ISECT_MT, C.ISECT_WATERTIGHT])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 3_039, 3_040, 3_041, 94_241, 97_279, 97_280, 194_559, 194_560, 194_561])
def test_hits_equal_the_binary_layouts(world, n, isect):
    _, scene, rays = world
    a = scene.trace_closest(rays[:n], isect, C.BVH_WIDE4)
    b = scene.trace_closest(rays[:n], isect, C.BVH_BINARY)
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("shift", [0, 4, 8])
def test_hit_buffers_at_any_word(world, shift):
    import torch

    ctx, scene, rays = world
    n = 1_000
    d_rays = torch.from_numpy(rays[:n]).cuda()
    buf = torch.full((n * 8 + 16,), 7.0, device="cuda")
    torch.cuda.synchronize()
    C.check(C.lib().illume_trace_closest_device(ctx.handle, scene.handle, d_rays.data_ptr(), n, C.ISECT_WATERTIGHT,
                                                C.BVH_WIDE4, buf.data_ptr() + shift))
    torch.cuda.synchronize()
    out = buf.cpu().numpy()
    got = out[shift // 4:shift // 4 + 8 * n].reshape(n, 8)
    ref = scene.trace_closest(rays[:n], C.ISECT_WATERTIGHT, C.BVH_BINARY)
    assert np.array_equal(got[:, 0], ref["t"]) and np.array_equal(got[:, 3:6].view(np.int32),
                                                                  np.stack([ref["inst"], ref["prim"], ref["sphere"]], 1))
    assert (got[:, 6:].view(np.int32) == 0).all()
    assert (out[:shift // 4] == 7.0).all() and (out[shift // 4 + 8 * n:] == 7.0).all()
