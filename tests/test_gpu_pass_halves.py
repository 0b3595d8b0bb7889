"""Without an environment a pass of 2^20 paths or more runs as two halves side by side. Asked
for one engine it runs whole; sums, sums of squares and ray counts are equal bit for bit, at
the size where the rule starts, odd path counts, one sample, several passes of which the
last is smaller, depths 1 to 25, and for next-event estimation, mediums and a second call."""
import numpy as np
import pytest

from illume_gb300 import _capi as C
from illume_gb300 import synth
from illume_gb300.api import Context, HostScene, Renderer
from illume_gb300.scenedata import Material, Mesh

pytestmark = pytest.mark.gpu


def scene(medium):
    s = synth.cornell_scene(64, 64)
    if medium:
        P, T = synth.displaced_icosphere(8, 3)
        med = s.add_medium(np.array([0.01, 0.08, 0.3]), 0.05, 0.7)
        glass = s.add_material(Material(C.MAT_REFRACTIVE, s.constant((1, 1, 1)), s.constant((1e-4,) * 3), ior=1.3, medium=med))
        M = np.zeros((3, 4), np.float32)
        M[:, :3], M[:, 3] = np.eye(3) * 120.0, (277.5, 140.0, 277.5)
        s.add_instance(s.add_mesh(Mesh(P, T)), glass, M)
    return s


@pytest.mark.parametrize("medium,estimator", [(False, 0), (False, 1), (True, 0)])
@pytest.mark.parametrize("isect", [C.ISECT_MT, C.ISECT_WATERTIGHT])
def test_halves_give_the_whole_pass(medium, estimator, isect):
    ctx = Context(0)
    sc = HostScene.from_data(ctx, scene(medium))

    def image(engines, w, h, spp, depth, per_pass):
        r = Renderer(ctx, sc, spp=spp, max_depth=depth, width=w, height=h, intersector=isect, estimator=estimator,
                     accum_mode=C.ACCUM_FP64, engines=engines, samples_per_pass=per_pass)
        first = r.render(sums=True)
        again = r.render(sums=True)
        r.close()
        assert np.array_equal(first["sum"], again["sum"], equal_nan=True)
        return first

    launches = set()
    for w, h, spp, depth, per_pass in ((1023, 1025, 1, 3, 0), (1024, 1024, 1, 4, 0), (1025, 1023, 1, 2, 0), (1031, 1021, 1, 1, 0),
                                       (333, 211, 15, 9, 0), (300, 301, 29, 25, 13)):
        a, b = image(0, w, h, spp, depth, per_pass), image(1, w, h, spp, depth, per_pass)
        assert a["stats"].rays == b["stats"].rays
        assert np.array_equal(a["sum"], b["sum"], equal_nan=True) and np.array_equal(a["sumsq"], b["sumsq"], equal_nan=True)
        launches.add(a["stats"].kernel_launches > b["stats"].kernel_launches)
    assert launches == {False, True}   # both routes were taken
    ctx.close()
