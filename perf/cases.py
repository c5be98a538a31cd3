"""What is timed: the work a user of convector_gb300 has it do.

A case names a path (its "kind"), the scene it runs on, sizes and options. The
scenes are the seeded ones of the benchmark (convector_gb300.scenes): the room
with a sphere (4,972 triangles), the displaced icosphere (81,930), the
random-walk tube (869,900) and the uneven sphere-and-box scenes. They stay
resident, as a renderer's or a server's do; rays, cameras, frames, requests and
meshes to build come from the seed.
"""

import functools
import math

import numpy as np
import torch

import convector_gb300 as cg
from convector_gb300 import scenes

FAR = 1.0e5
# Triangles, and boxes and triangles tested per ray on average by the nearest-hit
# traversal (the library's own counters), for the operation counts of work().
SCENES = {"room": (4972, 24.0, 2.5), "icosphere": (81932, 27.3, 1.93), "tube": (869900, 55.0, 4.0)}
BOX_FLOPS, TRIANGLE_FLOPS, SHADE_FLOPS = 24, 50, 300
RAYS_PER_PATH = 3.1  # a path of at most five bounces in these scenes
CENTER = np.array([0.0, 1.25, -2.0])


def listed():
    return [
        # A handful of picking or visibility rays from host arrays, as an editor
        # or a physics step asks for them: the latency of one call.
        {"name": "pick_1k", "kind": "pick", "scene": "icosphere", "rays": 1021, "traversal": "packet"},
        # The ray-cast workload of the benchmark, rays already on the device.
        {"name": "cast_icosphere_4m", "kind": "cast", "scene": "icosphere", "rays": 4194304, "traversal": "single"},
        # The reference's packets (the default traversal), a ragged count.
        {"name": "cast_room_packet_1m", "kind": "cast", "scene": "room", "rays": 1000003, "traversal": "packet"},
        # The interactive frame with the renderer's defaults.
        {"name": "frame_room", "kind": "frame", "scene": "room", "width": 1280, "height": 736, "rng": "group",
         "traversal": "packet"},
        # The same frame with the reference's own random stream (32x32 patches).
        {"name": "frame_room_patch", "kind": "frame", "scene": "room", "width": 1280, "height": 736, "rng": "patch",
         "traversal": "packet"},
        # A small preview.
        {"name": "frame_room_small", "kind": "frame", "scene": "room", "width": 320, "height": 184, "rng": "group",
         "traversal": "single"},
        # A full-HD frame of a mid-sized mesh.
        {"name": "frame_icosphere_hd", "kind": "frame", "scene": "icosphere", "width": 1920, "height": 1080,
         "rng": "group", "traversal": "single"},
        # Accumulative rendering of the large mesh, 16 samples, with the resolved image.
        {"name": "accumulate_tube_16", "kind": "accumulate", "scene": "tube", "width": 1280, "height": 736,
         "samples": 16, "traversal": "single"},
        # Many uneven scenes in one batch call, 4 samples each.
        {"name": "batch_32", "kind": "batch", "scenes": 32, "samples": 4},
        # A burst of render requests over the three resident scenes.
        {"name": "serve_16", "kind": "serve", "requests": 16},
        # One displayed frame: textures, 8-frame blend, median, sRGB.
        {"name": "display", "kind": "display", "width": 1280, "height": 736},
        # A new mesh admitted while serving: its BVH built on the device.
        {"name": "build_icosphere", "kind": "build", "mesh": "icosphere", "size": 6},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _frame_size(rng, widest):
    w = _log(rng, 160, widest)
    return w, max(90, min(1080, int(round(w * rng.uniform(0.5, 0.62)))))


def draw(rng):
    kind = rng.choice(["pick", "cast", "cast", "frame", "frame", "patch", "accumulate", "batch", "serve", "display",
                       "build"])
    scene = rng.choice(["room", "icosphere", "tube"])
    traversal = rng.choice(["single", "packet"])
    if kind == "pick":
        return {"kind": kind, "scene": scene, "rays": _log(rng, 1, 65536), "traversal": traversal}
    if kind == "cast":
        return {"kind": kind, "scene": scene, "rays": _log(rng, 65537, 4194304), "traversal": traversal}
    if kind == "frame":
        w, h = _frame_size(rng, 1920)
        return {"kind": kind, "scene": scene, "width": w, "height": h, "rng": "group", "traversal": traversal}
    if kind == "patch":
        w, h = _frame_size(rng, 1280)
        return {"kind": "frame", "scene": rng.choice(["room", "icosphere"]), "width": w, "height": h, "rng": "patch",
                "traversal": "packet"}
    if kind == "accumulate":
        w, h = _frame_size(rng, 1280)
        return {"kind": kind, "scene": scene, "width": w, "height": h, "samples": rng.randint(2, 16),
                "traversal": "single"}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 40), "samples": rng.randint(1, 6)}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(1, 16)}
    if kind == "display":
        w, h = _frame_size(rng, 1920)
        return {"kind": kind, "width": w, "height": h}
    mesh = rng.choice(["tube", "spheres"])  # size: rings of 512 triangles, triangles
    return {"kind": kind, "mesh": mesh, "size": _log(rng, 8, 320) if mesh == "tube" else _log(rng, 500, 20000)}


@functools.lru_cache(maxsize=None)
def _triangles(name):
    if name == "room":
        return scenes.room_sphere(obj=False)[0]
    if name == "icosphere":
        return scenes.displaced_icosphere(obj=False, light=True)[0]
    if name == "tube":
        return scenes.random_walk_tube(obj=False)[0]
    return scenes.spheres_and_boxes(*(int(v) for v in name.split("/")), obj=False)[0]


@functools.lru_cache(maxsize=None)
def _bvh(name):
    return cg.Bvh.build_device(_triangles(name))


@functools.lru_cache(maxsize=None)
def _scene(name):
    return cg.Scene(_bvh(name))


def _batch_plan(count):
    """Triangle counts (log-uniform 500..20,000) and image sizes of a batch's scenes, as in the benchmark."""
    rng = np.random.default_rng(3)
    counts = np.exp(rng.uniform(np.log(500), np.log(20000), count)).astype(int)
    sizes = [(320, 184), (640, 368), (1280, 736)]
    return ["%d/%d" % (c, 300009 + i) for i, c in enumerate(counts)], [sizes[i] for i in rng.integers(0, 3, count)]


def _serve_plan(count):
    """Scene, size and samples of each request: sizes log-uniform 320x184..1920x1080, 1..16 samples."""
    rng = np.random.default_rng(4)
    out = []
    for _ in range(count):
        w = int(round(np.exp(rng.uniform(np.log(320), np.log(1920)))))
        h = int(min(1080, max(184, round(w * 184 / 320))))
        out.append((int(rng.integers(0, 3)), w, h, int(rng.integers(1, 17))))
    return out


def _traversal(case):
    return cg.TRAVERSE_PACKET if case["traversal"] == "packet" else cg.TRAVERSE_SINGLE


def _rays(case, seed):
    # Origins uniform in the room, directions uniform on the sphere.
    return scenes.random_rays(case["rays"], seed=seed)


@functools.lru_cache(maxsize=None)
def _mesh(mesh, size):
    if mesh == "icosphere":
        return scenes.displaced_icosphere(subdivisions=size, obj=False)[0]
    if mesh == "tube":
        return scenes.random_walk_tube(rings=size, obj=False)[0]
    return scenes.spheres_and_boxes(size, 3, obj=False)[0]


def _instance(case, seed):
    # The mesh at another scale (a power of two, so that its tree has as many
    # nodes) with texture coordinates of its own.
    tris = _mesh(case["mesh"], case["size"]).copy()
    rng = np.random.default_rng(seed)
    f = tris.view(np.float32)
    f[:, :9] *= np.float32(2.0 ** int(rng.integers(-6, 7)))
    f[:, 9:15] = rng.random((f.shape[0], 6), dtype=np.float32)
    return tris


def prepare(case, seed):
    cg.lib()
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "pick":
        o, d = _rays(case, seed)
        return {"case": case, "scene": _scene(case["scene"]), "o": o, "d": d}
    if kind == "cast":
        o, d = _rays(case, seed)
        rays = torch.from_numpy(np.ascontiguousarray(np.concatenate([o.T, d.T]))).cuda()
        n = rays.shape[1]
        return {"case": case, "scene": _scene(case["scene"]), "rays": rays,
                "t": torch.empty(n, dtype=torch.float32, device="cuda"),
                "tri": torch.empty(n, dtype=torch.int32, device="cuda")}
    if kind in ("frame", "accumulate"):
        r = cg.Renderer(_scene(case["scene"]), case["width"], case["height"],
                        rng_order=cg.RNG_PATCH if case.get("rng") == "patch" else cg.RNG_GROUP,
                        traversal=_traversal(case))
        eye = (rng.uniform(-1.0, 1.0), rng.uniform(0.8, 1.6), 1.6)
        r.set_camera(scenes.default_camera(cg.Camera(), eye=eye))
        return {"case": case, "renderer": r, "frame": int(rng.integers(0, 1 << 20))}
    if kind == "batch":
        names, sizes = _batch_plan(case["scenes"])
        views = []
        for i, (w, h) in enumerate(sizes):
            cam = scenes.default_camera(cg.Camera(), eye=(rng.uniform(-1, 1), rng.uniform(0.8, 1.6), 1.6))
            views.append(cg.View(i, w, h, case["samples"], int(rng.integers(0, 1 << 20)), cam))
        batch = cg.Batch([_scene(n) for n in names], max_pixels=sum(w * h for w, h in sizes))
        return {"case": case, "batch": batch, "views": views}
    if kind == "serve":
        # The engine configuration of the benchmark's served section.
        server = cg.Server([_scene("room"), _scene("icosphere"), _scene("tube")], framebuffer_bytes=2 << 30,
                           refill_mode=cg.REFILL_ALL, deep_single_launch=1, samples_per_wave=16,
                           max_inflight_pixels=8 << 20)
        reqs = []
        for scene, w, h, spp in _serve_plan(case["requests"]):
            z, ph = rng.uniform(-1, 1), rng.uniform(0, 2 * np.pi)
            s = math.sqrt(1 - z * z)
            eye = CENTER + 3.0 * np.array([s * math.cos(ph), z, s * math.sin(ph)])
            cam = scenes.default_camera(cg.Camera(), eye=tuple(eye), target=tuple(CENTER))
            reqs.append((scene, w, h, spp, cam, int(rng.integers(0, 1 << 20))))
        return {"case": case, "server": server, "requests": reqs}
    if kind == "display":
        h, w = case["height"], case["width"]
        tex = [rng.integers(0, 256, (512, 512, 3), dtype=np.uint8) for _ in range(2)]
        # A rendered frame and its gbuffer words: texture coordinates, Fresnel
        # factor, and the texture index (0: no texture) in the top byte.
        rgba = rng.integers(0, 1 << 24, (h, w), dtype=np.uint32)
        gbuffer = rng.integers(0, 1 << 24, (h, w), dtype=np.uint32) | (rng.integers(0, 3, (h, w), dtype=np.uint32) << 24)
        return {"case": case, "display": cg.Display(w, h, tex[0], tex[1]), "rgba": rgba, "gbuffer": gbuffer}
    return {"case": case, "triangles": _instance(case, seed)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "pick":
        return state["scene"].intersect_nearest(state["o"], state["d"], far=FAR, traversal=_traversal(case))
    if kind == "cast":
        state["scene"].intersect_nearest_device(state["rays"], state["t"], state["tri"], far=FAR,
                                                traversal=_traversal(case),
                                                stream=torch.cuda.current_stream().cuda_stream)
        return state["t"], state["tri"]
    if kind == "frame":
        return state["renderer"].render_frame_u8(state["frame"])
    if kind == "accumulate":
        r = state["renderer"]
        r.clear_accumulator()
        gbuffer = r.accumulate_frames_f32(state["frame"], case["samples"], gbuffer=True)
        return r.resolve_u8(case["samples"]), gbuffer
    if kind == "batch":
        return state["batch"].render(state["views"])[0]
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(s, w, h, spp, cam, frame_base=f) for s, w, h, spp, cam, f in state["requests"]]
        return [server.wait(i)[1] for i in ids]
    if kind == "display":
        return state["display"].display_buffer(state["rgba"], state["gbuffer"])
    bvh = cg.Bvh.build_device(state["triangles"])
    return bvh.nodes, bvh.triangles, bvh.source_index


def _work_rays(scene, rays, shades):
    _, boxes, tris = SCENES[scene]
    return rays * (boxes * BOX_FLOPS + tris * TRIANGLE_FLOPS) + shades * SHADE_FLOPS


def _scene_bytes(triangles):
    # 48 bytes of geometry a triangle, and about one 32-byte node for two.
    return 64 * triangles


def work(case):
    kind = case["kind"]
    if kind in ("pick", "cast"):
        n = case["rays"]
        touched = min(_scene_bytes(SCENES[case["scene"]][0]), 1000 * n)
        return {"bytes": 32 * n + touched, "flops": _work_rays(case["scene"], n, 0)}
    if kind in ("frame", "accumulate"):
        px, spp = case["width"] * case["height"], case.get("samples", 1)
        rays = px * spp * RAYS_PER_PATH
        return {"bytes": 8 * px + _scene_bytes(SCENES[case["scene"]][0]), "flops": _work_rays(case["scene"], rays, rays)}
    if kind == "batch":
        names, sizes = _batch_plan(case["scenes"])
        px = sum(w * h for w, h in sizes)
        rays = px * case["samples"] * 2.0
        tris = sum(int(n.split("/")[0]) for n in names)
        return {"bytes": 4 * px + _scene_bytes(tris), "flops": _work_rays("room", rays, rays)}
    if kind == "serve":
        flops = px = 0
        for scene, w, h, spp in _serve_plan(case["requests"]):
            rays = w * h * spp * RAYS_PER_PATH
            flops += _work_rays(("room", "icosphere", "tube")[scene], rays, rays)
            px += w * h
        return {"bytes": 4 * px + sum(_scene_bytes(s[0]) for s in SCENES.values()), "flops": flops}
    if kind == "display":
        px = case["width"] * case["height"]
        return {"bytes": 44 * px, "flops": 200 * px}  # two inputs, the eight kept frames, one output
    n = {"icosphere": lambda s: 20 * 4 ** s, "tube": lambda s: 512 * s, "spheres": lambda s: s}[case["mesh"]](case["size"])
    return {"bytes": (64 + 64 + 4 + 32) * n, "flops": 300 * n * math.log2(n)}


def _brute_force(tris, o, d, far):
    """Distance to the nearest triangle of each ray, in 64 bits, against every triangle."""
    v = torch.from_numpy(tris.view(np.float32)[:, :9].astype(np.float64)).cuda()
    v0, v1, v2 = v[:, 0:3], v[:, 3:6], v[:, 6:9]
    e1, e2 = v0 - v2, v1 - v0
    n = torch.linalg.cross(e1, e2)
    o = torch.from_numpy(o.astype(np.float64)).cuda()
    d = torch.from_numpy(d.astype(np.float64)).cuda()
    t = torch.full((o.shape[0],), far, dtype=torch.float64, device="cuda")
    # dot(d, n), dot(v0 - o, n) and the two barycentric numerators, as matrix
    # products: dot(cross(d, v0 - o), e) = dot(d, cross(v0, e)) - dot(cross(d, o), e).
    step = max(1, (1 << 27) // v.shape[0])
    v0n = (v0 * n).sum(1)
    v0e1, v0e2 = torch.linalg.cross(v0, e1), torch.linalg.cross(v0, e2)
    for i in range(0, o.shape[0], step):
        oo, dd = o[i:i + step], d[i:i + step]
        m = torch.linalg.cross(dd, oo)
        den = 1.0 / (dd @ n.T)
        tt = (v0n - oo @ n.T) * den
        u = (dd @ v0e2.T - m @ e2.T) * den
        w = (dd @ v0e1.T - m @ e1.T) * den
        bad = ~((tt >= 0) & (u >= 0) & (w >= 0) & (u + w <= 1))
        t[i:i + step] = torch.minimum(t[i:i + step], tt.masked_fill_(bad, far).amin(1))
    return t


def exact(case, seed):
    # Images, gbuffer words, node arrays and indices are whole numbers; only the
    # queries' distances are computed numbers. 10^10 pairs of ray and triangle
    # take some seconds.
    if case["kind"] not in ("pick", "cast") or case["rays"] * SCENES[case["scene"]][0] > 10 ** 10:
        return None
    o, d = _rays(case, seed)
    return _brute_force(_triangles(case["scene"]), o, d, FAR), None
