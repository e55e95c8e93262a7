"""Performance cases of the path tracer: what programs have it do, by public entry points.

Each case is a dict of plain values with a "kind":

  frame   a resident scene and accumulator: reset, render, read the image (an interactive viewer, a
          turntable frame, a training-set view)
  call    TaichiRenderer.render() on a world: extraction, BVH build, render, image (a batch job's one call)
  build   a BVH build over resident triangles and a first set of ray queries (an edited mesh)
  query   ray queries against a built scene (picking, visibility, baking)
  atrous  the edge-aware a-trous filter, on device buffers or on host arrays
  infer   the learned denoiser on a rendered image's planes
  train   one gradient evaluation of the learned denoiser: features, forward, loss, backward
  obj     OBJ text to arrays
  batch   several scenes rendered as one batch

Sizes come from the workloads of this repository (the 1920x1080 64-spp displaced icosphere, the
256x256 Cornell box, the batched box scenes, the OBJ text, 128x128 training crops) or are generic.
"""
import ctypes
import math
import pathlib
import sys

import numpy as np
import torch

_PKG = str(pathlib.Path(__file__).resolve().parent.parent / "roxy-dcc_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import roxy_native as nat  # noqa: E402
import workloads  # noqa: E402
from core import Color, Vec3  # noqa: E402
from rendering.batch import BatchRenderer, Job  # noqa: E402
from rendering.denoise import edge_aware_denoise  # noqa: E402
from rendering.image import Image  # noqa: E402
from rendering.learned_denoiser import LAYERS, Denoiser, load_weights, macs_per_pixel  # noqa: E402
from rendering.taichi.extractor import build_device_scene  # noqa: E402
from rendering.taichi.trace import make_params  # noqa: E402
from rendering.taichi_renderer import TaichiRenderer  # noqa: E402
from scene import (Camera, Cube, Dielectric, Diffuse, Emissive, Glossy, ImageTexture, IndexedMesh,  # noqa: E402
                   Metal, Plane, SceneObject, Shape, Sphere, World)
from scene.io.obj_reader import parse_obj_bytes  # noqa: E402


def listed():
    return [
        # the final-quality frame of a large mesh: the framework's headline workload, the largest case
        dict(name="frame-1080p-64spp", kind="frame", scene="icosphere", size=7, w=1920, h=1080, spp=64, depth=12,
             lights="one", mis=False, passes=0, planes="radiance"),
        # the first image an interactive viewer shows after a camera move: latency and launches
        dict(name="preview-640x360-1spp", kind="frame", scene="icosphere", size=7, w=640, h=360, spp=1, depth=6,
             lights="one", mis=False, passes=0, planes="display"),
        # the small closed box with direct light at every bounce, filtered at the end
        dict(name="cornell-256-16spp-filtered", kind="frame", scene="cornell", size=0, w=256, h=256, spp=16, depth=8,
             lights="one", mis=False, passes=5, planes="radiance"),
        # an odd window over textures, glossy surfaces, planes and sphere lights, all lights sampled; the
        # guide planes are read as the learned denoiser's training views are
        dict(name="studio-413x307-8spp", kind="frame", scene="studio", size=0, w=413, h=307, spp=8, depth=6,
             lights="all", mis=True, passes=0, planes="all"),
        # one render call as a script makes it, world to image
        dict(name="call-960x540-16spp", kind="call", scene="icosphere", size=6, w=960, h=540, spp=16, depth=8,
             lights="one", passes=0),
        # a deformed mesh comes in: build its BVH, then pick into it
        dict(name="build-327k", kind="build", size=7, method="lbvh", leaf=4, rays=65536),
        # incoherent rays kept on the device, as a light or occlusion bake casts them
        dict(name="query-2m", kind="query", size=7, api="device", rays=2_000_003),
        # the filter in a frame loop that owns its buffers, at its largest common size
        dict(name="atrous-720p-5pass", kind="atrous", api="device", w=1280, h=720, radius=1, passes=5, guides=True),
        # the learned denoiser on a full-HD frame
        dict(name="infer-1080p", kind="infer", n=1, w=1920, h=1080),
        # a training step's gradients at the training configuration's crop and batch
        dict(name="train-16x128", kind="train", n=16, w=128, h=128),
        # an exported mesh file of tens of megabytes
        dict(name="obj-26mb", kind="obj", copies=4, size=6),
        # several users' scenes of mixed sizes in one batch
        dict(name="batch-8-scenes", kind="batch", scenes=8, tris=200_000, res=512, spp=16, depth=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "call", "build", "query", "query", "atrous", "infer", "train", "obj",
                       "batch"])
    if kind in ("frame", "call"):
        scene = rng.choice(["icosphere", "cornell", "studio", "boxes"])
        w, h = _log(rng, 64, 1920), _log(rng, 64, 1080)
        depth, lights = rng.randint(2, 16), rng.choice(["one", "all"])
        # closed scenes trace a ray and shadow rays at every bounce: bounded below the largest listed case
        rays = w * h * (4 if scene == "icosphere" else depth * (2 if lights == "one" else 4))
        spp = max(1, min(_log(rng, 1, 64), 100_000_000 // rays))
        c = dict(kind=kind, scene=scene,
                 size=rng.randint(4, 7) if scene == "icosphere" else _log(rng, 1000, 500_000) if scene == "boxes" else 0,
                 w=w, h=h, spp=spp, depth=depth, lights=lights,
                 passes=rng.choice([0, 0, 1, 5]))
        if kind == "frame":
            c.update(mis=rng.random() < 0.3, planes=rng.choice(["radiance", "display", "all"]))
        return c
    if kind == "build":
        return dict(kind=kind, size=rng.randint(3, 7), method=rng.choice(["lbvh", "lbvh", "morton"]),
                    leaf=rng.choice([2, 4, 8]), rays=_log(rng, 1000, 200_000))
    if kind == "query":
        return dict(kind=kind, size=rng.randint(3, 7), api=rng.choice(["device", "device", "closest", "any", "scene"]),
                    rays=_log(rng, 1000, 2_000_003))
    if kind == "atrous":
        api = rng.choice(["device", "host"])
        w, h = _log(rng, 33, 1920), _log(rng, 33, 1080)
        if api == "device":
            h = min(h, 1_048_576 // w)
        return dict(kind=kind, api=api, w=w, h=h, radius=rng.choice([1, 1, 1, 2, 3]), passes=rng.randint(1, 5),
                    guides=rng.random() < 0.8)
    if kind == "infer":
        return dict(kind=kind, n=1, w=4 * _log(rng, 16, 480), h=4 * _log(rng, 16, 270))
    if kind == "train":
        return dict(kind=kind, n=rng.randint(1, 16), w=4 * _log(rng, 8, 64), h=4 * _log(rng, 8, 64))
    if kind == "obj":
        return dict(kind=kind, copies=rng.randint(1, 6), size=rng.randint(3, 6))
    return dict(kind=kind, scenes=rng.randint(2, 12), tris=_log(rng, 2000, 300_000), res=rng.choice([96, 200, 256, 512]),
                spp=_log(rng, 1, 16), depth=rng.randint(2, 16))


# -- scenes ---------------------------------------------------------------------------------------
def _studio(w, h, rng):
    """Textured floor mesh, ground plane, glossy and metal spheres, a cube, two sphere lights, sky."""
    world = World(use_sky=True, background_color=Color(0.0, 0.0, 0.0))
    world.add_camera(Camera(position=Vec3(0.0, 1.1, 4.2), forward=Vec3(0, -0.2, -1), up=Vec3(0, 1, 0), fov=45,
                            width=w, height=h))
    tex = ImageTexture.from_array(rng.integers(0, 256, size=(64, 96, 3), dtype=np.uint8))
    pos = np.array([[-2, 0.01, -2], [2, 0.01, -2], [2, 0.01, 2], [-2, 0.01, 2]], np.float64)
    faces = np.array([[0, 2, 1], [0, 3, 2]], np.int32)
    uvs = np.array([[0, 0], [3, 0], [3, 3], [0, 3]], np.float64)
    rug = IndexedMesh(pos, faces, uvs=uvs, tri_uv_idx=faces, build_bvh=False)
    world.add_object(SceneObject(shapes=[Shape(rug, {"default": Diffuse(Color(0.9, 0.9, 0.9), albedo_texture=tex)})],
                                 name="rug"))
    world.add_object(SceneObject(shape=Plane(Vec3(0, 1, 0)), material=Diffuse(Color(0.5, 0.5, 0.45)), name="ground"))
    mats = [Glossy(Color(0.7, 0.2, 0.2), roughness=0.4), Metal(Color(0.9, 0.8, 0.6), roughness=0.1),
            Dielectric(Color(1.0, 1.0, 1.0), ior=1.5), Diffuse(Color(0.2, 0.5, 0.7))]
    for i in range(8):
        r = float(rng.uniform(0.15, 0.4))
        p = [float(rng.uniform(-1.6, 1.6)), r, float(rng.uniform(-1.5, 1.2))]
        world.add_object(SceneObject(shape=Sphere(r), material=mats[i % 4], translation=Vec3(*p), name=f"ball{i}"))
    world.add_object(SceneObject(shape=Cube(0.6), material=Diffuse(Color(0.6, 0.6, 0.2)),
                                 translation=Vec3(0.3, 0.3, -1.9), name="cube"))
    for i in range(2):
        world.add_object(SceneObject(shape=Sphere(0.2), material=Emissive(Color(1.0, 0.9, 0.8), intensity=12.0),
                                     translation=Vec3(-1.5 + 3.0 * i, 2.4, float(rng.uniform(-1, 1))), name=f"lamp{i}"))
    return world


def _world(case, seed):
    rng = np.random.default_rng(seed)
    w, h = case["w"], case["h"]
    if case["scene"] == "icosphere":
        return workloads.displaced_icosphere_scene(w, h, subdiv=case["size"], seed=seed)
    if case["scene"] == "cornell":
        return workloads.cornell_box(w, h, light_gap=float(rng.uniform(1e-3, 0.05)),
                                     light_size=float(rng.uniform(0.2, 0.35)))
    if case["scene"] == "boxes":
        return workloads.instanced_box_scene(case["size"], seed, w, h)
    return _studio(w, h, rng)


def _mesh(size, seed):
    """Displaced icosphere: float32 corner rows and the positions."""
    pos, faces = workloads.icosphere(size)
    pos = (pos * (1.0 + 0.05 * workloads.value_noise3(pos, seed + 1))[:, None]).astype(np.float32)
    return pos[faces[:, 0]], pos[faces[:, 1]], pos[faces[:, 2]]


def _rays(n, seed, mesh):
    """Rays aimed into the mesh from a shell, and a fifth of them leaving its surface."""
    rng = np.random.default_rng(seed + 17)
    unit = lambda k: (lambda v: v / np.linalg.norm(v, axis=1, keepdims=True))(  # noqa: E731
        rng.standard_normal((k, 3), dtype=np.float32))
    ro = unit(n) * rng.uniform(1.5, 3.5, (n, 1)).astype(np.float32)
    rd = unit(n) * rng.uniform(0.0, 1.1, (n, 1)).astype(np.float32) - ro
    k = n // 5
    tri = rng.integers(0, len(mesh[0]), k)
    ctr = (mesh[0][tri] + mesh[1][tri] + mesh[2][tri]) / np.float32(3.0)
    nrm = ctr / np.linalg.norm(ctr, axis=1, keepdims=True)
    ro[:k] = ctr + nrm * np.float32(1e-3)
    rd[:k] = nrm + unit(k) * np.float32(0.999)
    rd /= np.linalg.norm(rd, axis=1, keepdims=True)
    return np.ascontiguousarray(ro, np.float32), np.ascontiguousarray(rd, np.float32)


def _image_planes(n, h, w, seed):
    """A rendered image's planes: noisy radiance over smooth shading, guides with flat regions and edges."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    low = torch.rand((n, 12, max(2, h // 24), max(2, w // 24)), generator=g, device="cuda")
    up = torch.nn.functional.interpolate(low, size=(h, w), mode="nearest").permute(0, 2, 3, 1)
    albedo = (0.1 + 0.8 * up[..., 0:3]).contiguous()
    normal = torch.nn.functional.normalize(2.0 * up[..., 3:6] - 1.0, dim=-1).contiguous()
    depth = (1.0 + 4.0 * up[..., 6:7]).contiguous()
    noise = -torch.log1p(-0.999 * torch.rand((n, h, w, 1), generator=g, device="cuda"))
    radiance = (albedo * (0.2 + up[..., 7:10]) * (0.6 + 0.4 * noise)).contiguous()
    target = torch.log1p(albedo * (0.2 + up[..., 7:10])).contiguous()
    return radiance, albedo, normal, depth, target


# -- prepare --------------------------------------------------------------------------------------
def prepare(case, seed):
    s = {"case": case}
    kind = case["kind"]
    if kind == "frame":
        world = _world(case, seed)
        ds = build_device_scene(world)
        ds.use_lights(False)
        cam = workloads.camera_params(world, case["w"], case["h"])
        s.update(scene=ds, acc=nat.Accumulator(case["w"], case["h"]), spp=case["spp"], params=make_params(
            case["w"], case["h"], cam["fov_tan"], cam["aspect"], case["depth"], int(world.use_sky),
            0 if case["lights"] == "one" else 1, case["depth"] if case["scene"] != "icosphere" else 1, 10.0,
            list(world.background_color), cam["cam_pos"], cam["cam_fwd"], cam["cam_right"], cam["cam_up"], seed=seed,
            mis=case["mis"]))
        if case["passes"]:
            s["filter"] = nat.DenoiseParams(1, case["passes"], 0.08, 0.35, 0.20, 1.0, 0.8, 1, 1, 1, 1)
    elif kind == "call":
        image = Image(case["w"], case["h"])
        s.update(image=image, renderer=TaichiRenderer(
            _world(case, seed), image, None, samples=case["spp"], max_depth=case["depth"],
            direct_light_mode=case["lights"], denoise=case["passes"] > 0, denoise_passes=max(1, case["passes"]),
            seed=seed))
    elif kind == "build":
        mesh = _mesh(case["size"], seed)
        s.update(scene=nat.NativeScene(), rays=_rays(case["rays"], seed, mesh),
                 method=nat.RX_BVH_LBVH_SAH if case["method"] == "lbvh" else nat.RX_BVH_REFERENCE)
        s["scene"].set_triangles(*mesh)
    elif kind == "query":
        mesh = _mesh(case["size"], seed)
        sc = nat.NativeScene()
        sc.set_triangles(*mesh)
        sc.build_bvh()
        ro, rd = _rays(case["rays"], seed, mesh)
        n = case["rays"]
        s.update(scene=sc, ro=ro, rd=rd)
        if case["api"] == "device":
            s.update(ro=torch.from_numpy(ro).cuda(), rd=torch.from_numpy(rd).cuda(), n=n,
                     out=[torch.empty(n, dtype=torch.int32 if k == 1 else torch.float32, device="cuda")
                          for k in range(4)])
        elif case["api"] == "any":
            s["tmax"] = np.random.default_rng(seed + 5).uniform(0.5, 4.0, n).astype(np.float32)
    elif kind == "atrous":
        rad, alb, nrm, dep, _ = _image_planes(1, case["h"], case["w"], seed)
        if case["api"] == "device":
            pad = lambda t, w: torch.cat([t[0], w], dim=-1).contiguous()  # noqa: E731
            zero = torch.zeros_like(dep[0])
            s.update(color=pad(rad, zero), gn=pad(nrm, dep[0]), ga=pad(alb, zero))
            s["out"] = torch.empty_like(s["color"])
            g = 1 if case["guides"] else 0
            s["params"] = nat.DenoiseParams(case["radius"], case["passes"], 0.08, 0.35, 0.20, 1.0, 0.8, g, g, g, 0)
        else:
            s.update(color=rad[0].cpu().numpy(), normal=nrm[0].cpu().numpy(), albedo=alb[0].cpu().numpy(),
                     depth=dep[0, ..., 0].cpu().numpy())
    elif kind == "infer":
        s.update(net=Denoiser(weights=load_weights()), planes=_image_planes(case["n"], case["h"], case["w"], seed)[:4])
    elif kind == "train":
        s.update(net=Denoiser(seed=seed), planes=_image_planes(case["n"], case["h"], case["w"], seed))
    elif kind == "obj":
        s["text"] = workloads.obj_text(case["copies"], case["size"], seed)
    else:
        # the sizes of the jobs belong to the case; their scenes are the seed's
        specs = workloads.batch_specs(case["scenes"], 7, (1e3, case["tris"]),
                                      tuple(r for r in (case["res"] // 2, case["res"])),
                                      tuple(sorted({1, max(1, case["spp"] // 4), case["spp"]})), (2, case["depth"]))
        s["batch"] = BatchRenderer([
            Job(workloads.instanced_box_scene(j["n_tris"], 1000 * seed + i, j["width"], j["height"]), j["width"],
                j["height"], j["spp"], j["max_depth"], seed=1000 * seed + i) for i, j in enumerate(specs)])
    return s


# -- run ------------------------------------------------------------------------------------------
def _read(acc, planes):
    names = dict(radiance=nat.RX_ACC_RADIANCE, normal=nat.RX_ACC_NORMAL, albedo=nat.RX_ACC_ALBEDO,
                 depth=nat.RX_ACC_DEPTH, display=nat.RX_ACC_DISPLAY)
    keys = ("radiance", "albedo", "normal", "depth") if planes == "all" else (planes,)
    return {k: acc.read(names[k]) for k in keys}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "frame":
        acc = s["acc"]
        acc.reset()
        acc.render(s["scene"].native, s["params"], s["spp"])
        out = _read(acc, case["planes"])
        if case["passes"]:
            out["filtered"] = acc.denoise(s["filter"])
        return out
    if kind == "call":
        s["renderer"].render()
        return {"image": s["image"].pixels, "rays": s["renderer"].last_ray_count}
    if kind == "build":
        s["scene"].build_bvh(s["method"], case["leaf"])
        return s["scene"].trace_closest(*s["rays"])
    if kind == "query":
        if case["api"] == "closest":
            return s["scene"].trace_closest(s["ro"], s["rd"])
        if case["api"] == "any":
            return s["scene"].trace_any(s["ro"], s["rd"], s["tmax"])
        if case["api"] == "scene":
            return s["scene"].intersect(s["ro"], s["rd"])
        sc = s["scene"]
        sc.ctx.check(nat.lib().rx_trace_closest_device(
            sc.h, s["n"], *[ctypes.c_void_p(t.data_ptr()) for t in (s["ro"], s["rd"], *s["out"])]))
        return s["out"]
    if kind == "atrous":
        if case["api"] == "device":
            p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
            stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
            rc = nat.lib().rx_denoise_noalloc(case["h"], case["w"], p(s["color"]), p(s["gn"]), p(s["ga"]),
                                              ctypes.byref(s["params"]), p(s["out"]), stream)
            if rc:
                raise RuntimeError(nat.lib().rx_last_error(None).decode())
            return s["out"]
        g = dict(normal=s["normal"], albedo=s["albedo"], depth=s["depth"]) if case["guides"] else {}
        return edge_aware_denoise(s["color"], case["radius"], 0.08, 0.8, passes=case["passes"], **g)
    if kind == "infer":
        return s["net"].denoise(*s["planes"])
    if kind == "train":
        net, (rad, alb, nrm, dep, target) = s["net"], s["planes"]
        n, h, w = case["n"], case["h"], case["w"]
        for name, _, _, _ in LAYERS:
            net.dw[name].zero_()
            net.db[name].zero_()
        net.features(rad, alb, nrm, dep, n, h, w, train=True)
        net.forward(n, h, w, train=True)
        loss = net.loss(n, h, w, target)
        net.backward(n, h, w)
        return {"loss": loss, "dw": net.dw, "db": net.db}
    if kind == "obj":
        d = parse_obj_bytes(s["text"])
        return {"positions": d.positions, "normals": d.normals, "tri_pos": d.tri_pos_idx, "tri_nrm": d.tri_normal_idx,
                "group": d.tri_group_idx}
    b = s["batch"]
    for j in b.jobs:
        j.acc.reset()
    b.render()
    return [j.acc.read(nat.RX_ACC_RADIANCE) for j in b.jobs]


# -- work -----------------------------------------------------------------------------------------
def _ray_flops(tris):
    """A closest-hit query: about 2 log4(n) four-box tests (24 FMA each) and four triangle tests."""
    return 2.0 * max(1.0, math.log(max(tris, 4), 4)) * 48 + 4 * 45


def _scene_tris(case):
    return 20 * 4 ** case["size"] if case["scene"] == "icosphere" else max(case["size"], 36)


def work(case):
    kind = case["kind"]
    if kind in ("frame", "call"):
        px, tris = case["w"] * case["h"], _scene_tris(case)
        paths = px * case["spp"]
        planes = {"all": 40, "radiance": 12, "display": 12}[case.get("planes", "display")]
        # at least the camera rays, their shading (about 150 flops) and a running mean
        return {"bytes": 96.0 * tris + planes * px + (12 * px if case["passes"] else 0),
                "flops": paths * (_ray_flops(tris) + 200.0) + px * case["passes"] * 200.0}
    if kind == "build":
        n = 20 * 4 ** case["size"]
        return {"bytes": 36.0 * n + 48.0 * n + 32.0 * n + case["rays"] * 40.0, "flops": case["rays"] * _ray_flops(n)}
    if kind == "query":
        n = 20 * 4 ** case["size"]
        return {"bytes": case["rays"] * (52.0 if case["api"] == "scene" else 40.0) + 80.0 * n,
                "flops": case["rays"] * _ray_flops(n)}
    if kind == "atrous":
        px = case["w"] * case["h"]
        taps = (2 * case["radius"] + 1) ** 2
        return {"bytes": px * (64.0 if case["api"] == "device" else 52.0), "flops": px * case["passes"] * taps * 20.0}
    if kind in ("infer", "train"):
        px = case["n"] * case["h"] * case["w"]
        weights = sum(9 * cin * cout for _, cin, cout, _ in LAYERS)
        f = 2.0 * macs_per_pixel() * px
        if kind == "infer":
            return {"bytes": px * 52.0 + 2.0 * weights, "flops": f}
        return {"bytes": px * 52.0 + 6.0 * weights, "flops": 3.0 * f}
    if kind == "obj":
        v = 10 * 4 ** case["size"] + 2
        return {"bytes": case["copies"] * v * (60.0 + 48.0 + 2 * (60.0 + 28.0)), "flops": 0}
    return {"bytes": case["scenes"] * (case["res"] ** 2 * 12.0 + 96.0 * case["tris"] / 2),
            "flops": case["scenes"] * case["res"] ** 2 * max(1, case["spp"] // 3) * (_ray_flops(case["tris"]) + 200.0)}


# -- exact ----------------------------------------------------------------------------------------
def _reflect(i, n):
    if n == 1:
        return torch.zeros_like(i)
    i = torch.remainder(i, 2 * (n - 1))
    return torch.where(i >= n, 2 * (n - 1) - i, i)


def _atrous64(color, normal, albedo, depth, radius, passes, amount):
    h, w = color.shape[:2]
    two = lambda s: 2.0 * max(s * s, 1e-8)  # noqa: E731
    ys, xs = torch.arange(h, device=color.device), torch.arange(w, device=color.device)
    cur = color
    for i in range(passes):
        num, den = torch.zeros_like(color), torch.zeros((h, w, 1), dtype=torch.float64, device=color.device)
        for dy in range(-radius, radius + 1):
            for dx in range(-radius, radius + 1):
                yy, xx = _reflect(ys + (dy << i), h)[:, None], _reflect(xs + (dx << i), w)[None, :]
                at = lambda t: t[yy, xx]  # noqa: E731
                e = ((at(cur) - cur) ** 2).sum(-1, keepdim=True) / two(0.08)
                if normal is not None:
                    e = e + ((at(normal) - normal) ** 2).sum(-1, keepdim=True) / two(0.35)
                    e = e + ((at(albedo) - albedo) ** 2).sum(-1, keepdim=True) / two(0.20)
                    e = e + (at(depth) - depth) ** 2 / two(1.0)
                wt = torch.exp(-e) / (1.0 + dx * dx + dy * dy)
                num += at(cur) * wt
                den += wt
        cur = num / den.clamp_min(1e-8)
    return color * (1.0 - amount) + cur * amount


def _network64(net, planes, weights):
    """The network in 64 bits on the bf16 weights: (log-space output, log1p radiance)."""
    F = torch.nn.functional
    rad, alb, nrm, dep = (t.double() for t in planes)
    base = torch.log1p(rad.clamp_min(0.0))
    dep = dep.clamp_min(0.0)
    x = torch.cat([base, alb, nrm, dep / (1.0 + dep)], dim=-1)
    x = F.pad(x, (0, 6)).permute(0, 3, 1, 2)

    def c(name, x):
        _, cin, cout, relu = next(layer for layer in LAYERS if layer[0] == name)
        wt = weights[name].reshape(cout, 3, 3, cin).permute(0, 3, 1, 2)
        y = F.conv2d(x, wt, net.b32[name].double(), padding=1) if not wt.requires_grad else \
            F.conv2d(x, wt, weights["b_" + name], padding=1)
        return torch.relu(y) if relu else y

    up = lambda t: F.interpolate(t, scale_factor=2, mode="nearest")  # noqa: E731
    s1 = c("e1b", c("e1a", x))
    s2 = c("e2b", c("e2a", F.avg_pool2d(s1, 2)))
    m = c("e3b", c("e3a", F.avg_pool2d(s2, 2)))
    m = c("d2b", c("d2a", torch.cat([up(m), s2], 1)))
    m = c("d1b", c("d1a", torch.cat([up(m), s1], 1)))
    return c("head", m).permute(0, 2, 3, 1)[..., :3], base


def _closest64(ro, rd, mesh):
    """Nearest t, u, v of each ray over all triangles in 64 bits (a miss: 1e9, 0, 0)."""
    v0, v1, v2 = (torch.from_numpy(m).cuda().double() for m in mesh)
    e1, e2 = v1 - v0, v2 - v0
    dot = lambda a, b: (a * b).sum(-1)  # noqa: E731
    ts, us, vs = [], [], []
    step = max(1, 16_000_000 // len(v0))
    for i in range(0, len(ro), step):
        o, d = (torch.from_numpy(a[i:i + step]).cuda().double()[:, None, :] for a in (ro, rd))
        h = torch.linalg.cross(d.expand(-1, len(v0), -1), e2[None].expand(d.shape[0], -1, -1))
        det = dot(e1[None], h)
        f = 1.0 / torch.where(det.abs() > 1e-8, det, torch.ones_like(det))
        sv = o - v0[None]
        u = f * dot(sv, h)
        q = torch.linalg.cross(sv, e1[None].expand_as(sv))
        v = f * dot(d, q)
        t = f * dot(e2[None], q)
        ok = (det.abs() > 1e-8) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > 1e-3)
        t = torch.where(ok, t, torch.full_like(t, 1e9))
        best, k = t.min(dim=1)
        pick = lambda a: torch.where(best < 1e9, a.gather(1, k[:, None])[:, 0], torch.zeros_like(best))  # noqa: E731
        ts.append(best)
        us.append(pick(u))
        vs.append(pick(v))
    return torch.cat(ts), torch.cat(us), torch.cat(vs)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("build", "query") and case.get("api", "device") in ("device", "closest"):
        if case["rays"] * 20 * 4 ** case["size"] > 2e9:
            return None  # brute force over all triangles takes too long
        mesh = _mesh(case["size"], seed)
        t, u, v = _closest64(*_rays(case["rays"], seed, mesh), mesh)
        return [t, None, u, v]
    if kind == "atrous":
        rad, alb, nrm, dep, _ = (t[0].double() for t in _image_planes(1, case["h"], case["w"], seed))
        if not case["guides"]:
            nrm = alb = dep = None
        r = _atrous64(rad, nrm, alb, dep, case["radius"], case["passes"], 0.8)
        return torch.nn.functional.pad(r, (0, 1)) if case["api"] == "device" else r
    if kind == "infer":
        net = Denoiser(weights=load_weights())
        y, base = _network64(net, _image_planes(case["n"], case["h"], case["w"], seed)[:4],
                             {k: v.double() for k, v in net.w16.items()})
        return torch.expm1(y + base).clamp_min(0.0)
    if kind == "train":
        net = Denoiser(seed=seed)
        *planes, target = _image_planes(case["n"], case["h"], case["w"], seed)
        wts = {k: v.double().requires_grad_() for k, v in net.w16.items()}
        wts.update({"b_" + k: v.double().requires_grad_() for k, v in net.b32.items()})
        y, base = _network64(net, planes, wts)
        diff = (y + base - target.double()).abs()
        (diff.sum() / diff.numel()).backward()
        return {"loss": diff.detach().sum().reshape(1), "dw": {k: wts[k].grad for k in net.w16},
                "db": {k: wts["b_" + k].grad for k in net.w16}}
    if kind == "obj":
        lines = workloads.obj_text(case["copies"], case["size"], seed).split(b"\n")
        rows = lambda key: np.array(b" ".join(x[len(key):] for x in lines if x.startswith(key)).split(),  # noqa: E731
                                    dtype=np.float64).reshape(-1, 3)
        return {"positions": rows(b"v "), "normals": rows(b"vn "), "tri_pos": None, "tri_nrm": None, "group": None}
    return None
