"""Small passes run as one path-kernel launch (up to 2^18 paths) and larger ones hand the
rest of their paths over once at most 2^17 rays are left. The binary layout runs the
wavefront stages alone; its images and ray counts are the yardstick, bit for bit, on both
sides of each limit, for depths at which nothing, something or everything is handed over."""
import ctypes

import numpy as np
import pytest

from illume_gb300 import _capi as C
from illume_gb300 import synth
from illume_gb300.api import Context, HostScene, Renderer, Server
from illume_gb300.scenedata import Material, Mesh

pytestmark = pytest.mark.gpu


def scene(kind):
    if kind == "ground":
        return synth.traversal_scene(tris=2_000, env_size=(64, 32))
    s = synth.cornell_scene(64, 64)
    if kind == "medium":
        P, T = synth.displaced_icosphere(8, 3)
        med = s.add_medium(np.array([0.01, 0.08, 0.3]), 0.05, 0.7)
        glass = s.add_material(Material(C.MAT_REFRACTIVE, s.constant((1, 1, 1)), s.constant((1e-4,) * 3), ior=1.3, medium=med))
        M = np.zeros((3, 4), np.float32)
        M[:, :3], M[:, 3] = np.eye(3) * 120.0, (277.5, 140.0, 277.5)
        s.add_instance(s.add_mesh(Mesh(P, T)), glass, M)
    return s


@pytest.mark.parametrize("kind,estimator", [("ground", 0), ("ground", 1), ("cornell", 0), ("cornell", 1), ("medium", 0)])
@pytest.mark.parametrize("isect", [C.ISECT_MT, C.ISECT_WATERTIGHT])
def test_images_equal_the_wavefronts(kind, estimator, isect):
    ctx = Context(0)
    sc = HostScene.from_data(ctx, scene(kind))

    def image(bvh, w, h, spp, depth):
        r = Renderer(ctx, sc, spp=spp, max_depth=depth, width=w, height=h, intersector=isect, estimator=estimator,
                     accum_mode=C.ACCUM_FP64, bvh_kind=bvh)
        out = r.render(sums=True)
        again = r.render(sums=True)
        assert np.array_equal(out["sum"], again["sum"], equal_nan=True) and out["stats"].rays == again["stats"].rays
        r.close()
        return out["sum"], out["sumsq"], out["stats"].rays

    # 1 path; a partial warp; 2^18 paths exactly and one row more; passes that shrink to 2^17 late or never
    for w, h, spp, depth in ((1, 1, 1, 1), (7, 5, 1, 6), (512, 512, 1, 3), (512, 513, 1, 2), (512, 513, 1, 3),
                             (300, 301, 5, 5), (512, 512, 2, 9), (640, 480, 3, 17)):
        a, b = image(C.BVH_WIDE4, w, h, spp, depth), image(C.BVH_BINARY, w, h, spp, depth)
        assert a[2] == b[2]
        assert np.array_equal(a[0], b[0], equal_nan=True) and np.array_equal(a[1], b[1], equal_nan=True)
    ctx.close()


def test_jobs_of_different_depths_share_a_table():
    ctx = Context(0)
    scenes = [HostScene.from_data(ctx, scene(k)) for k in ("ground", "cornell", "medium")]
    jobs = []
    for j, (w, h, spp, depth) in enumerate(((33, 21, 3, 1), (64, 64, 2, 7), (50, 40, 4, 16), (128, 96, 9, 4), (400, 300, 3, 12))):
        p = scenes[j % 3].default_params(spp, depth)
        p.width, p.height, p.seed, p.job = w, h, 5, j
        jobs.append((scenes[j % 3], p))
    srv = Server(ctx, lanes=1)
    ids = [srv.submit(*job) for job in jobs]
    srv.run()
    for i, (sc, p) in zip(ids, jobs):
        got = srv.poll(i)
        p.bvh_kind = C.BVH_BINARY
        r = Renderer(ctx, sc, params=p)
        ref = r.render()
        assert np.array_equal(got["mean"], ref["mean"], equal_nan=True) and got["stats"].rays == ref["stats"].rays
        r.close()
    ctx.close()


@pytest.mark.parametrize("kind", ["ground", "medium"])
def test_overlapping_engines_hand_over_too(kind):
    ctx = Context(0)
    sc = HostScene.from_data(ctx, scene(kind))
    out = []
    for bvh, engines in ((C.BVH_BINARY, 1), (C.BVH_WIDE4, 2), (C.BVH_WIDE4, 4)):
        r = Renderer(ctx, sc, spp=8, max_depth=11, width=512, height=300, accum_mode=C.ACCUM_FP64, bvh_kind=bvh,
                     engines=engines)
        o = r.render(sums=True)
        out.append((o["sum"], o["stats"].rays))
        r.close()
    for s, n in out[1:]:
        assert n == out[0][1] and np.array_equal(s, out[0][0], equal_nan=True)
    ctx.close()
