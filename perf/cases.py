"""The renderer's work as its users call it: renders from a thumbnail to a full traversal
step, both estimators, all three accumulation modes, both triangle tests, the allocation-free
frame loop, batches of ray queries from host and from device buffers, and a served mix of
requests. Every case goes through the public entry points (illume_gb300.api, and the C-ABI
calls that have no Python wrapper).

A case's inputs follow from its seed: the meshes' displacement, the camera's place, the
materials, the rays and the Philox key of the render.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from illume_gb300 import _capi as C
from illume_gb300 import synth
from illume_gb300.api import Context, HostScene, Renderer, Server
from illume_gb300.scenedata import Material, Mesh, SceneData, Texture

ISECT = {"mt": C.ISECT_MT, "watertight": C.ISECT_WATERTIGHT}
ACCUM = {"fp32": C.ACCUM_FP32, "kahan": C.ACCUM_KAHAN, "fp64": C.ACCUM_FP64}
TONE = {"linear": C.TONE_LINEAR, "reinhard": C.TONE_REINHARD, "filmic": C.TONE_FILMIC, "uncharted": C.TONE_UNCHARTED}
BVH = {"wide4": C.BVH_WIDE4, "binary": C.BVH_BINARY}


def _render(name, scene, tris, width, height, spp, depth, isect="watertight", accum="fp32", tone="linear", nee=False,
            exact_hg=False, sums=False):
    return dict(name=name, kind="render", scene=scene, tris=tris, width=width, height=height, spp=spp, depth=depth,
                isect=isect, accum=accum, tone=tone, nee=nee, exact_hg=exact_hg, sums=sums)


def listed():
    return [
        # a thumbnail while a scene is edited: one sample per pixel, all of it latency
        _render("thumbnail", "cornell", 12, 64, 48, 1, 8),
        # a frame loop that may not allocate: a small image at two samples per pixel
        dict(name="frame_loop", kind="noalloc", scene="ground", tris=20_000, width=200, height=150, spp=2, depth=10,
             isect="watertight"),
        # an interactive preview: one sample of every pixel of a 720p frame
        _render("preview_720p", "mixed", 100_000, 1280, 720, 1, 10, tone="filmic"),
        # the Cornell box, a whole small render
        _render("cornell", "cornell", 12, 256, 256, 64, 8, isect="mt"),
        # an odd frame of a scene with vertex normals, texture coordinates and bitmaps
        _render("textured_odd", "textured", 30_011, 333, 219, 24, 15, accum="kahan", tone="reinhard"),
        # the triangle-heavy traversal step: the largest render
        _render("traversal", "ground", 100_000, 1024, 1024, 128, 25, isect="mt"),
        # subsurface: a long random walk in a medium behind a smooth dielectric, sums read back
        _render("subsurface", "medium", 200_000, 480, 360, 16, 50, accum="fp64", exact_hg=True, sums=True),
        # many large instanced meshes whose trees outgrow the caches
        _render("instanced", "instanced", 2_000_000, 512, 512, 32, 12),
        # next-event estimation under an environment map with a sun
        _render("light_sampling", "ground", 100_000, 512, 512, 32, 25, isect="mt", nee=True),
        # a picking query: some rays from host memory
        dict(name="pick", kind="trace", scene="ground", tris=20_000, rays=1_003, isect="watertight", bvh="wide4",
             device=False),
        # a visibility bake: incoherent rays that are already on the device
        dict(name="bake", kind="trace", scene="instanced", tris=500_000, rays=3_000_017, isect="watertight",
             bvh="wide4", device=True),
        # a render server with requests of different sizes over two scenes
        dict(name="served", kind="serve", tris=60_000, requests=8, side=384, spp=48, depth=15, isect="watertight"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render"] * 7 + ["noalloc", "trace", "trace", "serve"])
    isect = rng.choice(["mt", "watertight"])
    if kind == "noalloc":
        w, h = _log(rng, 32, 255), _log(rng, 32, 255)
        return dict(kind=kind, scene=rng.choice(["cornell", "ground", "mixed"]), tris=_log(rng, 500, 100_000), width=w,
                    height=h, spp=rng.randint(1, 4), depth=rng.randint(3, 15), isect=isect)
    if kind == "trace":
        device = rng.random() < 0.6
        return dict(kind=kind, scene=rng.choice(["ground", "mixed", "instanced"]), tris=_log(rng, 2_000, 500_000),
                    rays=_log(rng, 100, 3_000_000 if device else 300_000), isect=isect,
                    bvh=rng.choice(["wide4", "wide4", "binary"]), device=device)
    if kind == "serve":
        return dict(kind=kind, tris=_log(rng, 5_000, 100_000), requests=rng.randint(2, 9), side=rng.randint(96, 512),
                    spp=rng.randint(8, 64), depth=rng.randint(8, 20), isect=isect)
    scene = rng.choice(["cornell", "ground", "mixed", "textured", "medium", "instanced"])
    # pixels x samples over the whole range; scenes with longer paths stay below the largest case
    top = 4_000_000 if scene == "medium" else 40_000_000
    paths = _log(rng, 2_000, top)
    pixels = min(paths, _log(rng, 2_000, 1_200_000))
    aspect = math.exp(rng.uniform(-0.5, 0.7))
    width = max(16, int(math.sqrt(pixels * aspect)))
    height = max(16, pixels // width)
    tris = _log(rng, 200_000, 2_000_000) if scene == "instanced" else _log(rng, 1_000, 200_000)
    case = _render("", scene, 12 if scene == "cornell" else tris, width, height, max(1, paths // (width * height)),
                   rng.randint(3, 25) if scene != "medium" else rng.randint(8, 50), isect=isect,
                   accum=rng.choice(["fp32", "fp32", "kahan", "fp64"]), tone=rng.choice(sorted(TONE)),
                   nee=scene != "medium" and rng.random() < 0.2, exact_hg=rng.random() < 0.5, sums=rng.random() < 0.2)
    del case["name"]
    return case


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _context() -> Context:
    # one context (one stream) per process, as a program that renders keeps one; calls of
    # the allocation-free entry point have to share a stream
    return Context(0)


@functools.lru_cache(maxsize=None)
def _sphere(freq: int):
    return synth.icosphere(freq)


@functools.lru_cache(maxsize=None)
def _sky(width: int, height: int):
    return synth.environment_map(1, width, height)


def _blob(tris: int, rng, amp: float = 0.15):
    """A displaced sphere of about `tris` triangles: ten random waves over the unit sphere."""
    P, T = _sphere(synth.freq_for_tris(tris))
    r = np.ones(len(P))
    for o in range(10):
        k = rng.normal(size=3) * (2.0 + 1.5 * o)
        r += amp / (1.0 + 0.6 * o) * 0.5 * np.sin(P @ k + rng.uniform(0.0, 2.0 * math.pi))
    return (P * r[:, None]).astype(np.float32), T


def _look(s, rng, pos, target, spread):
    pos = np.asarray(pos, np.float64) + rng.uniform(-spread, spread, 3)
    s.camera_transform = synth.lookat(pos, target)
    s.camera_fov, s.camera_dof, s.camera_aperture = 40.0, 1.0, 0.0


def _scene(kind: str, tris: int, rng) -> SceneData:
    if kind == "cornell":
        s = synth.cornell_scene(256, 256)
        s.camera_transform = s.camera_transform.copy()
        s.camera_transform[:, 3] += rng.uniform(-15.0, 15.0, 3).astype(np.float32)
        return s
    if kind == "medium":
        # a dielectric around a dense medium in the Cornell box
        s = synth.cornell_scene(256, 256, spheres=False)
        P, T = _blob(tris, rng)
        med = s.add_medium(np.array([0.01, 0.08, 0.3]), 1.0, 0.7)
        glass = s.add_material(Material(C.MAT_REFRACTIVE, s.constant((1, 1, 1)), s.constant((1e-4,) * 3), ior=1.3,
                                        medium=med))
        M = np.zeros((3, 4), np.float32)
        M[:, :3] = np.eye(3) * 120.0
        M[:, 3] = (277.5, 140.0, 277.5)
        s.add_instance(s.add_mesh(Mesh(P, T)), glass, M)
        s.camera_transform = s.camera_transform.copy()
        s.camera_transform[:, 3] += rng.uniform(-15.0, 15.0, 3).astype(np.float32)
        return s
    s = SceneData()
    if kind == "ground":
        # a rough metal shape over a checkered lambert ground, lit by the sky
        P, T = _blob(tris, rng)
        metal = s.add_material(Material(C.MAT_ROUGHCONDUCTOR, s.constant((0, 0, 0)), s.constant((0.2,) * 3),
                                        eta=synth.GOLD_ETA, k=synth.GOLD_K, distribution=C.DIST_GGX))
        checker = s.add_texture(Texture(C.TEX_CHECKERBOARD, color=(0.8,) * 3, off=(0.2,) * 3, scale=(16.0, 16.0)))
        lambert = s.add_material(Material(C.MAT_LAMBERT, checker, s.constant((1e-4,) * 3)))
        s.add_instance(s.add_mesh(Mesh(P, T)), metal)
        GP, GT, GUV = synth.quad(20.0, -1.2)
        s.add_instance(s.add_mesh(Mesh(GP, GT, texcoords=GUV)), lambert)
        _look(s, rng, (0.0, 0.8, -4.2), (0.0, -0.15, 0.0), 0.3)
        s.ray_bias = 1e-4
    elif kind == "textured":
        # vertex normals and texture coordinates, an HDR and an 8-bit bitmap, glass and plastic spheres
        P, T = _blob(tris, rng)
        N = P / np.linalg.norm(P, axis=1, keepdims=True)
        UV = np.stack([np.arctan2(N[:, 2], N[:, 0]) / (2 * math.pi) + 0.5, np.arccos(np.clip(N[:, 1], -1, 1)) / math.pi],
                      axis=1).astype(np.float32)
        hdr = np.ones((67, 131, 4), np.float32)
        hdr[..., :3] = rng.uniform(0.1, 0.9, (67, 131, 3))
        ldr = np.full((64, 96, 4), 255.0, np.float32)
        ldr[..., :3] = rng.integers(30, 230, (64, 96, 3))
        body = s.add_material(Material(C.MAT_LAMBERT, s.add_texture(Texture(C.TEX_BITMAP, scale=(3.0, 2.0), texels=hdr)),
                                       s.constant((1e-4,) * 3)))
        floor = s.add_material(Material(C.MAT_PLASTIC, s.add_texture(Texture(C.TEX_BITMAP, scale=(4.0, 4.0), texels=ldr,
                                                                            hdr=0)), s.constant((1e-4,) * 3), ior=1.5))
        s.add_instance(s.add_mesh(Mesh(P, T, normals=N.astype(np.float32), texcoords=UV)), body)
        GP, GT, GUV = synth.quad(20.0, -1.2)
        s.add_instance(s.add_mesh(Mesh(GP, GT, texcoords=GUV)), floor)
        s.add_sphere((1.6, -0.7, -0.6), 0.5, s.add_material(
            Material(C.MAT_REFRACTIVE, s.constant((1, 1, 1)), s.constant((1e-4,) * 3), ior=1.5)))
        s.add_sphere((-1.7, -0.6, 0.2), 0.6, s.add_material(
            Material(C.MAT_ROUGHREFLECTIVE, s.constant((0.9, 0.8, 0.7)), s.constant((0.3,) * 3), ior=1.5)))
        _look(s, rng, (0.0, 0.9, -4.6), (0.0, -0.2, 0.0), 0.3)
        s.ray_bias = 1e-4
    else:
        # "mixed": a handful of instances of two meshes; "instanced": sixteen meshes of their own
        count = 5 if kind == "mixed" else 16
        meshes = [s.add_mesh(Mesh(*_blob(max(20, tris // (2 if kind == "mixed" else count)), rng)))
                  for _ in range(2 if kind == "mixed" else count)]
        for i in range(count):
            M = np.zeros((3, 4))
            M[:, :3] = synth.random_rotation(rng) * (rng.uniform(0.6, 1.6) if kind == "mixed" else 1.0)
            M[:, 3] = rng.uniform(-3.0, 3.0, 3) if kind == "mixed" else (3.0 * (i % 4) - 4.5, 0.0, 3.0 * (i // 4) - 4.5)
            s.add_instance(meshes[i % len(meshes)], synth.mixed_material(s, rng), M.astype(np.float32))
        if kind == "mixed":
            _look(s, rng, (0.0, 3.0, -9.0), (0.0, 0.0, 0.0), 0.5)
        else:
            _look(s, rng, (0.0, 8.0, -14.0), (0.0, 0.0, 0.0), 0.5)
        s.ray_bias = 1e-3
    size = (2048, 1024) if kind in ("ground", "instanced") else (512, 256)
    s.env_tex = s.add_texture(Texture(C.TEX_BITMAP, texels=_sky(*size), hdr=1))
    return s


def _rays(kind: str, n: int, rng) -> np.ndarray:
    """Rays from a shell around the scene toward points inside it: unordered, some missing."""
    extent = {"ground": 1.3, "mixed": 4.0, "instanced": 6.0}[kind]
    flat = np.array([1.0, 0.3 if kind == "instanced" else 1.0, 1.0])
    o = rng.normal(size=(n, 3)).astype(np.float32)
    o *= (rng.uniform(1.5, 3.0, n) * extent / np.linalg.norm(o, axis=1)).astype(np.float32)[:, None]
    d = (rng.uniform(-extent, extent, (n, 3)) * flat).astype(np.float32) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    out = np.zeros((n, 8), np.float32)
    out[:, :3], out[:, 4:7] = o, d
    return out


def _params(scene, case, seed, **over):
    p = scene.default_params(case["spp"], case["depth"])
    p.width, p.height = case["width"], case["height"]
    p.intersector = ISECT[case["isect"]]
    p.seed, p.job = seed & 0x7FFFFFFF, 1
    for k, v in over.items():
        setattr(p, k, v)
    return p


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    ctx = _context()
    kind = case["kind"]
    if kind == "serve":
        scenes = [HostScene.from_data(ctx, _scene(k, case["tris"], rng)) for k in ("ground", "mixed")]
        jobs = []
        sizes = np.random.default_rng(case["side"])   # the case names the mix; the seed makes its scenes and samples
        for j in range(case["requests"]):
            f = math.exp(sizes.uniform(math.log(0.25), 0.0))
            w, h = max(16, int(case["side"] * f)), max(16, int(case["side"] * f * 0.75))
            req = dict(case, width=w, height=h, spp=max(1, int(case["spp"] * sizes.uniform(0.2, 1.0))))
            sc = scenes[int(sizes.integers(2))]
            jobs.append((sc, _params(sc, req, seed, job=j)))
        return dict(kind=kind, server=Server(ctx), jobs=jobs)
    data = _scene(case["scene"], case["tris"], rng)
    scene = HostScene.from_data(ctx, data)
    if kind == "trace":
        rays = _rays(case["scene"], case["rays"], rng)
        st = dict(kind=kind, ctx=ctx, scene=scene, isect=ISECT[case["isect"]], bvh=BVH[case["bvh"]], n=case["rays"],
                  device=case["device"], rays=rays)
        if case["device"]:
            st["rays"] = torch.from_numpy(rays).cuda()
            st["hits"] = torch.zeros((case["rays"], 8), dtype=torch.float32, device="cuda")
            torch.cuda.synchronize()
        return st
    if kind == "noalloc":
        sums = torch.zeros((case["width"] * case["height"], 3), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        return dict(kind=kind, ctx=ctx, scene=scene, params=_params(scene, case, seed), sums=sums)
    p = _params(scene, case, seed, accum_mode=ACCUM[case["accum"]], tonemapper=TONE[case["tone"]],
                estimator=C.ESTIMATOR_NEE if case["nee"] else C.ESTIMATOR_REFERENCE, exact_hg=int(case["exact_hg"]))
    return dict(kind=kind, renderer=Renderer(ctx, scene, params=p), sums=case["sums"])


def run(state):
    kind = state["kind"]
    if kind == "render":
        out = state["renderer"].render(mean=True, sums=state["sums"], rgb8=True)
        res = dict(mean=out["mean"], rgb8=out["rgb8"], rays=int(out["stats"].rays))
        if state["sums"]:
            res["sum"], res["sumsq"] = out["sum"], out["sumsq"]
        return res
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(scene, params) for scene, params in state["jobs"]]
        srv.run()
        done = [srv.poll(i, rgb8=True) for i in ids]
        return [dict(mean=d["mean"], rgb8=d["rgb8"], rays=int(d["stats"].rays)) for d in done]
    if kind == "noalloc":
        ctx = state["ctx"]
        C.check(C.lib().illume_render_noalloc(ctx.handle, state["scene"].handle, C.ctypes.byref(state["params"]),
                                              state["sums"].data_ptr()))
        return state["sums"]
    if state["device"]:
        C.check(C.lib().illume_trace_closest_device(state["ctx"].handle, state["scene"].handle,
                                                    state["rays"].data_ptr(), state["n"], state["isect"], state["bvh"],
                                                    state["hits"].data_ptr()))
        hits = state["hits"]
        return dict(tuv=hits[:, :3], ids=hits[:, 3:6].view(torch.int32))
    return state["scene"].trace_closest(state["rays"], state["isect"], state["bvh"])


# ---------------------------------------------------------------- what a pass cannot do without
# closest-hit and shadow queries per path of a scene kind, at the depths used here
_RAYS_PER_PATH = {"cornell": 4.8, "ground": 2.1, "mixed": 1.4, "textured": 2.0, "medium": 12.0, "instanced": 1.5}


def _tree_bytes(tris):
    return 48 * tris + 128 * (tris // 6 + 1)


def _query_flops(tris):
    # two child boxes per binary level (15 operations each) and two triangles (50 each)
    return 30.0 * math.log2(max(tris, 2)) + 100.0


def work(case):
    kind = case["kind"]
    tris = case["tris"] + 2
    if kind == "trace":
        touched = min(_tree_bytes(tris), 200 * case["rays"])
        return {"bytes": 64 * case["rays"] + touched, "flops": case["rays"] * _query_flops(tris)}
    if kind == "serve":
        paths = case["requests"] * case["side"] ** 2 * 0.75 * 0.35 * case["spp"] * 0.6
        rays = paths * 1.75
        return {"bytes": int(2 * _tree_bytes(tris) + paths / case["spp"] * 15 * 2), "flops": rays * (_query_flops(tris) + 200.0)}
    npix = case["width"] * case["height"]
    rays = npix * case["spp"] * min(_RAYS_PER_PATH[case["scene"]], case["depth"])
    if kind == "noalloc":
        return {"bytes": min(_tree_bytes(tris), int(200 * rays)) + 12 * npix, "flops": rays * (_query_flops(tris) + 200.0)}
    out = npix * (15 + (48 if case["sums"] else 0))
    queries = rays * (2.0 if case["nee"] else 1.0)
    return {"bytes": min(_tree_bytes(tris), int(200 * rays)) + out, "flops": queries * _query_flops(tris) + rays * 200.0}


# ---------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    """Closest hits by testing every triangle in 64 bits; the other cases follow random paths
    whose 64-bit form is a renderer of its own."""
    if case["kind"] != "trace" or case["rays"] * float(case["tris"]) > 6e9:
        return None
    rng = np.random.default_rng(seed)
    s = _scene(case["scene"], case["tris"], rng)
    rays = torch.from_numpy(_rays(case["scene"], case["rays"], rng)).cuda().double()
    n = len(rays)
    best = torch.full((n,), math.inf, dtype=torch.float64, device="cuda")
    bu, bv = torch.zeros_like(best), torch.zeros_like(best)
    for (mi, _, _, inv, _) in s.instances:
        m = s.meshes[mi]
        A = torch.from_numpy(np.asarray(inv, np.float64)).cuda()
        o = rays[:, :3] @ A[:, :3].T + A[:, 3]
        d = rays[:, 4:7] @ A[:, :3].T
        V = torch.from_numpy(m.positions[m.tris].astype(np.float64)).cuda()
        v0, e1, e2 = V[:, 0], V[:, 1] - V[:, 0], V[:, 2] - V[:, 0]
        nrm = torch.linalg.cross(e1, e2)
        step = max(1, int(2e7) // len(V))
        for a in range(0, n, step):
            oo, dd = o[a:a + step], d[a:a + step]
            # t = (v0 - o).n / d.n; barycentrics from the edge determinants
            det = -(dd @ nrm.T)
            t = (oo @ nrm.T - (v0 * nrm).sum(1)) / det
            x = torch.linalg.cross(oo, dd)                      # o x d
            v0e1, v0e2 = torch.linalg.cross(e1, v0), torch.linalg.cross(e2, v0)
            u = ((x @ e2.T) - dd @ v0e2.T) / det
            v = (dd @ v0e1.T - (x @ e1.T)) / det
            t = torch.where((u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0), t, torch.inf)
            tm, k = t.min(1)
            r = torch.arange(len(oo), device="cuda")
            closer = tm < best[a:a + step]
            best[a:a + step] = torch.where(closer, tm, best[a:a + step])
            bu[a:a + step] = torch.where(closer, u[r, k], bu[a:a + step])
            bv[a:a + step] = torch.where(closer, v[r, k], bv[a:a + step])
    miss = torch.isinf(best)
    best = torch.where(miss, torch.full_like(best, float(np.finfo(np.float32).max)), best)
    if case["device"]:
        return dict(tuv=torch.stack([best, bu, bv], dim=1), ids=None)
    out = dict(t=best, u=bu, v=bv)
    out = {k: v.cpu().numpy() for k, v in out.items()}
    return dict(out, inst=None, prim=None, sphere=None)
