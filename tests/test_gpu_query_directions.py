"""Batch queries take directions as given, of any length. The 4-wide layout's hits equal the
binary layout's for directions near the largest float, whose reciprocals are subnormal: a
box test that flushed them to zero would lose the boxes such a ray enters. (Longest
component c x 2^126 with c in (1, 2), another below 2^126; triangles 0.1 across, so that no
product of the triangle tests overflows; origins 3 units away, so that distances are normal
numbers.)"""
import numpy as np
import pytest

from illume_gb300 import _capi as C
from illume_gb300 import synth
from illume_gb300.api import HostScene
from illume_gb300.scenedata import Material, Mesh, SceneData

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("instances", [1, 3, 17])
@pytest.mark.parametrize("isect", [C.ISECT_MT, C.ISECT_WATERTIGHT])
def test_long_directions(ctx, instances, isect):
    rng = np.random.default_rng(instances)
    s = SceneData()
    lambert = s.add_material(Material(C.MAT_LAMBERT, s.constant((0.5,) * 3), s.constant((1e-4,) * 3)))
    mesh = s.add_mesh(Mesh(*synth.icosphere(16)))
    for i in range(instances):
        M = np.eye(3, 4, dtype=np.float32)
        M[:, 3] = rng.uniform(-0.3, 0.3, 3) * (i > 0)
        s.add_instance(mesh, lambert, M)
    scene = HostScene.from_data(ctx, s)
    n = 2000
    target = rng.normal(size=(n, 3))
    target *= 0.6 / np.linalg.norm(target, axis=1, keepdims=True)
    for scale in (1.0, 2.0**60, 2.0**126):
        d = rng.uniform(0.1, 0.6, (n, 3)) * rng.choice([-1.0, 1.0], (n, 3))
        d[np.arange(n), rng.integers(3, size=n)] = rng.uniform(1.1, 1.6, n) * rng.choice([-1.0, 1.0], n)
        o = target - 3.0 * d
        rays = np.zeros((n, 8), np.float32)
        rays[:, :3], rays[:, 4:7] = o, d * scale
        a = scene.trace_closest(rays, isect, C.BVH_WIDE4)
        b = scene.trace_closest(rays, isect, C.BVH_BINARY)
        assert (b["inst"] >= 0).all()   # every ray passes through a body it starts outside of
        for key in b:
            assert np.array_equal(a[key], b[key]), (scale, key, int((a["inst"] != b["inst"]).sum()))
