"""Workloads of the indirect-lighting path as a renderer runs it.

Every case goes through the package's public entry points (Pipeline, Batch and
the C ABI behind them), on one stream that all contexts of the process share,
as an engine has one render stream. A case names sizes and options; the seed
places the boxes, camera and lights (or draws the samples).

`exact` restates the path in 64-bit torch, from the same inputs, without the
library: decisions that the path defines in binary32 (which cell a pixel lands
in, which voxels a face covers) are taken in binary32 here too.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from dynamicradiancevolume_gb300 import abi, batch, check, load, pipeline, surrogate

# ---------------------------------------------------------------- the cases


def _frame(name, width, height, boxes, voxels, lights, rsm, lod, cascades, cav, sh, steps, **more):
    case = {"name": name, "kind": "frame", "width": width, "height": height, "boxes": boxes, "voxels": voxels,
            "lights": lights, "rsm": rsm, "lod": lod, "shadow_lod": 0, "cascades": cascades, "cascade_size": 0.25,
            "cav": cav, "sh": sh, "steps": steps, "transition": 2.0, "bf16": False, "targets16": False,
            "shadow": True, "specular": 0, "surrogate": False, "max_caches": 262144}
    case.update(more)
    return case


def listed():
    return [
        # The repository's small configuration (a preview, a probe update, a
        # test scene): every launch is short, so launches and their gaps count.
        _frame("frame_small", 256, 256, 12, 64, 1, 32, 0, 1, 32, 1, 16, cascade_size=2.0, transition=0.0,
               max_caches=65536),
        # A window of a size nobody planned for: no side is a multiple of a
        # tile, two lights, shadow blocks of four VPLs.
        _frame("frame_window", 1013, 571, 31, 128, 2, 256, 2, 3, 32, 2, 24, shadow_lod=1, max_caches=65536),
        # The headline frame in the reference's render targets (SRGB8 diffuse,
        # 16-bit RSM, RGBA16F out) with 16-bit storage: what a game ships.
        _frame("frame_1080p", 1920, 1080, 64, 256, 1, 512, 3, 4, 32, 2, 32, bf16=True, targets16=True),
        # Production settings in full precision: three lights, 12288 VPLs.
        _frame("frame_production", 1920, 1080, 64, 256, 3, 512, 3, 4, 32, 2, 32),
        # Fine cascades: about 22 thousand caches, millions of shadow cones.
        _frame("frame_fine", 1920, 1080, 64, 256, 1, 512, 3, 4, 128, 2, 32, bf16=True, targets16=True),
        # Glossy surfaces: the per-cache specular envmaps of the reference's size.
        _frame("frame_specular", 1600, 900, 64, 256, 1, 512, 3, 4, 32, 2, 32, targets16=True, specular=16),
        # The learned visibility in place of the cones (shipped weights), at a
        # size of the batched configuration.
        _frame("frame_surrogate", 768, 768, 40, 128, 2, 512, 4, 4, 32, 2, 32, bf16=True, targets16=True,
               surrogate=True, max_caches=65536),
        # INDIRECT_SHADOW off: the cheap quality setting.
        _frame("frame_unshadowed", 1280, 720, 64, 128, 1, 512, 3, 4, 32, 2, 32, shadow=False, max_caches=16384),
        # A mesh scene's inputs: G-buffer, RSM and voxels rasterised from
        # triangles, walls of two triangles beside finely divided objects.
        {"name": "mesh_inputs", "kind": "mesh", "width": 1280, "height": 720, "boxes": 64, "divide": 10,
         "divide_room": 1, "voxels": 256, "lights": 1, "rsm": 512, "lod": 3},
        # The ground truth a scene is checked against: every VPL at every pixel.
        {"name": "ground_truth", "kind": "brute", "width": 960, "height": 540, "boxes": 64, "lights": 1, "rsm": 512,
         "lod": 3, "materials": False},
        # A training step of the visibility network at the trainer's batch.
        {"name": "train_step", "kind": "train", "samples": 4096},
        # Several scenes of uneven sizes (the batch's menus) as one graph.
        {"name": "batch_scenes", "kind": "batch", "scenes": 8, "first": 0, "streams": 4},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["mesh", "brute", "train", "batch"])
    if kind == "train":
        return {"kind": "train", "samples": _spread(rng, 200, 16384)}
    if kind == "batch":
        while True:  # the menus' scenes differ by a factor of a hundred: no more work than the listed batch
            case = {"kind": "batch", "scenes": rng.randint(2, 8), "first": rng.randint(0, 40),
                    "streams": rng.choice([1, 2, 4])}
            if work(case)["flops"] <= work({"kind": "batch", "scenes": 8, "first": 0})["flops"]:
                return case
    boxes, width = rng.randint(6, 64), _spread(rng, 160, 1920)
    height = max(90, min(1080, int(width * rng.uniform(0.5, 1.0))))
    if kind == "mesh":
        return {"kind": "mesh", "width": min(width, 1280), "height": min(height, 720), "boxes": boxes,
                "divide": rng.randint(1, 10), "divide_room": rng.randint(1, 6), "voxels": rng.choice([64, 128, 256]),
                "lights": 1, "rsm": rng.choice([128, 256, 512]), "lod": 2}
    if kind == "brute":
        return {"kind": "brute", "width": min(width, 960), "height": min(height, 540), "boxes": boxes,
                "lights": 1, "rsm": 256, "lod": rng.choice([2, 3, 4]), "materials": rng.random() < 0.3}
    special = rng.choice(["", "", "", "", "specular", "surrogate", "unshadowed"])
    cav = _spread(rng, 12, 128) if not special else rng.choice([24, 32, 48])
    lights, lod = (1, 3) if cav > 40 else rng.choice([(1, 3), (2, 3), (3, 3), (1, 4), (2, 4)])
    bf16 = rng.random() < 0.5
    case = _frame("", width, height, boxes, rng.choice([64, 128, 256]), lights, rng.choice([256, 512]), lod,
                  rng.randint(1, 4), cav, rng.choice([1, 2, 2]), rng.randint(8, 32), bf16=bf16,
                  targets16=bf16 or special != "" or rng.random() < 0.3, shadow_lod=rng.choice([0, 0, 0, 1]),
                  transition=rng.choice([0.0, 1.5, 2.0]), shadow=special != "unshadowed",
                  specular=rng.choice([8, 16]) if special == "specular" else 0, surrogate=special == "surrogate",
                  max_caches=131072 if cav > 40 else 32768)
    del case["name"]
    return case


# ---------------------------------------------------------------- what a program has in hand
_streams = {}


def _render_stream():
    """The process's one render stream."""
    dev = torch.cuda.current_device()
    if dev not in _streams:
        _streams[dev] = torch.cuda.Stream(dev)
    return _streams[dev]


def _workload(case):
    brute_or_mesh = case["kind"] in ("mesh", "brute")
    return pipeline.Workload(
        "case", case["width"], case["height"], case["boxes"], case.get("voxels", 64), case["lights"], case["rsm"],
        case["lod"], case.get("shadow_lod", 0), case.get("cascades", 1), case.get("cascade_size", 2.0),
        case.get("cav", 32), case.get("sh", 1), case.get("steps", 32), case.get("max_caches", 4096),
        cascade_transition=case.get("transition", 0.0), indirect_shadow=int(case.get("shadow", not brute_or_mesh)),
        precision=abi.PRECISION_BF16 if case.get("bf16") else abi.PRECISION_FP32,
        visibility=abi.VISIBILITY_SURROGATE if case.get("surrogate") else abi.VISIBILITY_CONE,
        specular_envmap_size=case.get("specular", 0))


def _lit_scene(workload, seed):
    """The first scene of the seed's series whose lights reach into the room
    (a spot light that hangs right above a box lights only the box's top,
    which nothing the camera sees faces): its seed."""
    k = np.arange(48)
    phi, tilt = k * 2.399963, np.radians(26.0) * np.sqrt((k + 0.5) / 48)
    for s in range(seed * 16, seed * 16 + 16):
        hf = pipeline.host_frame(workload, s)
        lo = np.array([hf.boxes[b].min[:] for b in range(hf.scene.n_boxes)], np.float64)
        hi = np.array([hf.boxes[b].max[:] for b in range(hf.scene.n_boxes)], np.float64)
        reach = []
        for light in hf.light_descs:
            o, d = np.array(light.position[:], np.float64), np.array(light.direction[:], np.float64)
            u = np.cross(d, [1.0, 0.0, 0.0])
            u /= np.linalg.norm(u)
            v = np.cross(d, u)
            rays = np.cos(tilt)[:, None] * d + np.sin(tilt)[:, None] * (np.cos(phi)[:, None] * u + np.sin(phi)[:, None] * v)
            t0, t1 = (lo[None] - o) / rays[:, None], (hi[None] - o) / rays[:, None]
            near, far = np.minimum(t0, t1).max(-1), np.maximum(t0, t1).min(-1)
            hit = np.where((near <= far) & (near > 0), near, np.inf)
            hit[:, 0] = far[:, 0]  # box 0 is the room, seen from inside
            reach.append(hit.min(1).mean())
        if np.mean(reach) >= 0.4:
            break
    return s


def _pipeline(case, seed):
    w = _workload(case)
    hf = pipeline.host_frame(w, _lit_scene(w, seed))
    t16 = case.get("targets16", False)
    if t16:
        hf.config.output_format = abi.OUTPUT_RGBA16F
    hf.config.surrogate_conf_threshold = 0.5
    p = pipeline.Pipeline(hf, albedo_format=abi.ALBEDO_SRGB8 if t16 else abi.ALBEDO_F32X3,
                          rsm_format=abi.RSM_F16 if t16 else abi.RSM_F32)
    p.stream = _render_stream()
    check(p.lib.drv_set_stream(p.ctx, C.c_void_p(p.stream.cuda_stream)), p.ctx)
    return p


def _srgb_encode(lin):
    cs = torch.where(lin <= 0.0031308, lin * 12.92, 1.055 * lin.clamp(min=1e-9) ** (1 / 2.4) - 0.055)
    return (cs * 255.0).round().clamp(0, 255).to(torch.uint8)


def _fill_inputs(p, seed):
    """The frame's G-buffer and RSMs, as the renderer's earlier passes leave them."""
    p.raycast_inputs()
    torch.cuda.synchronize()
    if p.albedo8 is not None:
        p.albedo8.copy_(_srgb_encode(p.albedo.double()))
        for l in range(p.hf.workload.n_lights):
            p.rsm_flux16[l].copy_(p.rsm_flux[l])
            p.rsm_dls16[l].copy_(p.rsm_dls[l])
    g = torch.Generator(device=p.device)
    g.manual_seed(seed)
    p.rough_metal.copy_(torch.randint(0, 256, p.rough_metal.shape, generator=g, device=p.device, dtype=torch.uint8))
    torch.cuda.synchronize()


class _Buffer:
    """A buffer of a pipeline's context; keeps the pipeline (and so the memory) alive."""

    def __init__(self, p, ptr, numel, typestr):
        self.owner = p
        self.__cuda_array_interface__ = {"shape": (numel,), "typestr": typestr, "data": (int(ptr), False),
                                         "version": 3, "strides": None}


def _view(p, ptr, numel, typestr):
    """A buffer of p's context as a tensor (no copy)."""
    return torch.as_tensor(_Buffer(p, ptr, numel, typestr), device="cuda")


def _box_mesh(hf, divide, divide_room, device):
    """The scene's boxes as an indexed triangle mesh: every face a grid of divide^2 quads."""
    pos, idx, alb, base = [], [], [], 0
    for b in range(hf.scene.n_boxes):
        box = hf.boxes[b]
        lo, hi = np.array(box.min[:], np.float64), np.array(box.max[:], np.float64)
        k = divide_room if box.inward else divide
        s = np.linspace(0.0, 1.0, k + 1)
        u, v = (q.ravel() for q in np.meshgrid(s, s))
        j, i = (q.ravel() for q in np.meshgrid(np.arange(k), np.arange(k)))
        corner = i * (k + 1) + j
        quads = np.concatenate([np.stack([corner, corner + 1, corner + k + 2], 1),
                                np.stack([corner, corner + k + 2, corner + k + 1], 1)])
        for axis in range(3):
            for side in range(2):
                p = np.empty(((k + 1) ** 2, 3))
                p[:, axis] = hi[axis] if side else lo[axis]
                a1, a2 = (axis + 1) % 3, (axis + 2) % 3
                p[:, a1], p[:, a2] = lo[a1] + u * (hi[a1] - lo[a1]), lo[a2] + v * (hi[a2] - lo[a2])
                pos.append(p)
                idx.append(quads + base)
                alb.append(np.tile(np.array(box.albedo[:], np.float32), (len(quads), 1)))
                base += len(p)
    t = lambda a, dt: torch.from_numpy(np.ascontiguousarray(np.concatenate(a).astype(dt))).to(device)
    return t(pos, np.float32), t(idx, np.int32), t(alb, np.float32)


def _train_data(case, seed):
    """Feature rows of the 17-input set (positions, normal, mostly empty
    opacity samples) and cone visibilities (many fully lit or fully dark),
    and a trainer some steps into its run."""
    n = case["samples"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    r = lambda *s: torch.rand(s, generator=g, device="cuda")
    X = torch.zeros((n, abi.SURROGATE_INPUTS), device="cuda")
    X[:, 0:6] = r(n, 6)
    X[:, 6:9] = torch.nn.functional.normalize(r(n, 3) - 0.5, dim=1)
    X[:, 9:17] = (r(n, 8) - 0.6).clamp(min=0.0) * r(n, 8)
    X[:, 31] = 1.0
    Y = ((r(n) * 2.0 - 0.5).clamp(0.0, 1.0) * torch.exp(-2.0 * X[:, 9:17].sum(1))).contiguous()
    params = torch.from_numpy(surrogate.init_params(seed % 1000)).cuda()
    m = (r(params.numel()) - 0.5) * 2e-3
    v = r(params.numel()) * 1e-5 + 1e-6
    return X, Y, params, m, v


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        p = _pipeline(case, seed)
        if case["surrogate"]:
            surrogate.upload(p, surrogate.load_params(), surrogate.load_features())
        _fill_inputs(p, seed)
        counter = _view(p, p.buffers().counter, 4, "<i4")
        return {"kind": kind, "p": p, "counter": counter}
    if kind == "brute":
        p = _pipeline(case, seed)
        _fill_inputs(p, seed)
        p.prepare_and_extract()
        rm = (p.rough_metal.float() / 255.0).contiguous() if case["materials"] else None
        torch.cuda.synchronize()
        return {"kind": kind, "p": p, "rough_metal": rm, "out": torch.zeros_like(p.out)}
    if kind == "mesh":
        p = _pipeline(case, seed)
        pos, idx, alb = _box_mesh(p.hf, case["divide"], case["divide_room"], p.device)
        mesh = abi.DrvMesh(pos.data_ptr(), None, alb.data_ptr(), idx.data_ptr(), pos.shape[0], idx.shape[0])
        gout = abi.DrvGBufferOut(p.depth.data_ptr(), p.normal16.data_ptr(), p.normal32.data_ptr(), p.albedo.data_ptr())
        routs = [abi.DrvRSMOut(p.rsm_flux[l].data_ptr(), p.rsm_normal[l].data_ptr(), p.rsm_dls[l].data_ptr())
                 for l in range(case["lights"])]
        b, n = p.buffers(), case["voxels"]
        texels = sum((n >> l) ** 3 for l in range(1, b.n_voxel_levels))
        outs = {"depth": p.depth, "normal16": p.normal16, "normal": p.normal32, "albedo": p.albedo,
                "flux": p.rsm_flux, "rsm_normal": p.rsm_normal, "depth_lin_sq": p.rsm_dls,
                "voxels": _view(p, b.voxel_bits, n ** 3 // 32, "<i4"), "mips": _view(p, b.voxel_mips[1], texels, "<f4")}
        torch.cuda.synchronize()
        return {"kind": kind, "p": p, "mesh": mesh, "gout": gout, "routs": routs, "keep": (pos, idx, alb), "outs": outs}
    if kind == "train":
        X, Y, params, m, v = _train_data(case, seed)
        scratch = torch.empty(load().drv_surrogate_train_scratch_floats(case["samples"]), device="cuda")
        return {"kind": kind, "X": X, "Y": Y, "params": params, "m": m, "v": v, "scratch": scratch,
                "loss": torch.zeros(2, device="cuda"), "step": 500}
    specs = [(w, _lit_scene(w, seed * 8 + i))
             for i, (w, _) in enumerate(batch.batch_workloads(case["scenes"], case["first"]))]
    scenes = batch.make_scenes(specs)
    return {"kind": kind, "scenes": scenes, "batch": batch.Batch(scenes, case["streams"], _render_stream())}


# ---------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind == "frame":
        s["p"].frame()
        return {"radiance": s["p"].out, "counter": s["counter"]}
    if kind == "brute":
        s["p"].bruteforce(s["out"], s["rough_metal"])
        return s["out"]
    if kind == "mesh":
        p, lib, hf = s["p"], s["p"].lib, s["p"].hf
        w = hf.workload
        check(lib.drv_raster_gbuffer(p.ctx, C.byref(s["mesh"]), C.byref(hf.camera), C.byref(hf.frame), w.width,
                                     w.height, C.byref(s["gout"])), p.ctx)
        for l, out in enumerate(s["routs"]):
            check(lib.drv_raster_rsm(p.ctx, C.byref(s["mesh"]), C.byref(hf.lights[l]), C.byref(out)), p.ctx)
        p.voxelize_triangles(s["keep"][0], s["keep"][1])
        return s["outs"]
    if kind == "train":
        ptr = lambda t: C.c_void_p(t.data_ptr())
        s["step"] += 1
        check(load().drv_surrogate_train_step(
            ptr(s["X"]), ptr(s["Y"]), s["X"].shape[0], ptr(s["params"]), ptr(s["m"]), ptr(s["v"]), ptr(s["scratch"]),
            s["step"], 1e-3, 0.03, 1e-4, ptr(s["loss"]), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return {"params": s["params"], "m": s["m"], "v": s["v"], "loss": s["loss"]}
    s["batch"].launch()
    return [sc.pipe.out for sc in s["scenes"]]


# ---------------------------------------------------------------- what a pass cannot do without
def _frame_work(case):
    px = case["width"] * case["height"]
    t16, vpls = case.get("targets16", False), case["lights"] * (case["rsm"] >> case["lod"]) ** 2
    blocks = vpls >> (2 * case.get("shadow_lod", 0))
    # Depth and normal, diffuse, materials; the RSMs; the output.
    bytes_ = px * (8 + (3 if t16 else 12) + (2 if case["specular"] else 0) + (8 if t16 else 12))
    bytes_ += case["lights"] * case["rsm"] ** 2 * (4 + (10 if t16 else 20))
    # Typical allocation: four tenths of a cascade's face in caches. Every
    # VPL of every cache is tested (5 flops), a tenth of the pairs are lit
    # (94), their blocks traced (a trilinear tap of 14 flops per step, about
    # half the steps); eight corners of SH products per pixel.
    caches = 0.4 * case["cascades"] * case["cav"] ** 2
    flops = caches * (5 * vpls + 9.4 * vpls) + px * (8 * 6 * (9 if case["sh"] == 2 else 4) + 60)
    if case["shadow"]:
        flops += caches * 0.1 * blocks * (20736 if case["surrogate"] else 14 * case["steps"] / 2)
    if case["specular"]:
        flops += px * 8 * 24 + caches * 0.1 * vpls * 30
    return {"bytes": bytes_, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "frame":
        return _frame_work(case)
    if kind == "brute":
        px, vpls = case["width"] * case["height"], case["lights"] * (case["rsm"] >> case["lod"]) ** 2
        return {"bytes": px * (20 + 12 + (8 if case["materials"] else 0)) + vpls * 48,
                "flops": px * vpls * (60 if case["materials"] else 34)}
    if kind == "mesh":
        px, texels, n = case["width"] * case["height"], case["lights"] * case["rsm"] ** 2, case["voxels"]
        tris = 12 * (case["boxes"] * case["divide"] ** 2 + case["divide_room"] ** 2)
        verts = 6 * (case["boxes"] * (case["divide"] + 1) ** 2 + (case["divide_room"] + 1) ** 2)
        # The mesh, the G-buffer (32 B a pixel), the RSM (24 B), the voxel
        # bits, their mips and the two sampling copies.
        return {"bytes": tris * 24 + verts * 12 + px * 32 + texels * 24 + n ** 3 * (1 / 8 + 4 / 7 + 1 + 16 / 7),
                "flops": 3 * tris * 100 + (px + texels) * 100}
    if kind == "train":
        n, weights = case["samples"], abi.SURROGATE_PARAMS
        return {"bytes": n * (abi.SURROGATE_INPUTS + 1) * 4 + weights * 4 * 6, "flops": 6.0 * n * weights}
    total = {"bytes": 0.0, "flops": 0.0}
    for w, _ in batch.batch_workloads(case["scenes"], case["first"]):
        one = _frame_work({"width": w.width, "height": w.height, "lights": w.n_lights, "rsm": w.rsm_resolution,
                           "lod": w.rsm_read_lod, "cascades": w.n_cascades, "cav": w.cav_res, "sh": w.sh_order,
                           "steps": w.max_cone_steps, "shadow": True, "surrogate": True, "specular": 0})
        total = {k: total[k] + one[k] for k in total}
    return total


# ---------------------------------------------------------------- 64-bit values
PI = 3.14159265358979323846


def _f64(x):
    return torch.tensor(list(x), dtype=torch.float64, device="cuda")


def _unpack_normal(n16):
    a, b = n16[..., 0].double() * (PI / 32768.0), n16[..., 1].double() / 32768.0
    s = torch.sqrt((1.0 - b * b).clamp(min=0.0))
    return torch.nn.functional.normalize(torch.stack([torch.cos(a) * s, torch.sin(a) * s, b], -1), dim=-1)


def _pack_normal(n):
    phi = torch.where(n[..., 0] == 0, torch.sign(n[..., 1]) * (PI / 2), torch.atan2(n[..., 1], n[..., 0]))
    v = torch.stack([phi / PI * 32768.0, n[..., 2] * 32768.0], -1).trunc()
    return v.clamp(-32768, 32767)


def _rsm_level(p, l, light):
    """(flux, normal, (d, d^2)) chain of light l down to the level the shadow blocks read."""
    flux = (p.rsm_flux16 or p.rsm_flux)[l].double()
    dls = (p.rsm_dls16 or p.rsm_dls)[l].double()
    chain = [(flux, p.rsm_normal[l], dls)]
    depth = int(math.log2(light.rsm_render_resolution // light.rsm_read_resolution)) + int(light.indirect_shadow_lod)
    for _ in range(depth):
        f, n, d = chain[-1]
        quads = lambda t: t[0::2, 0::2] + t[0::2, 1::2] + t[1::2, 0::2] + t[1::2, 1::2]
        ns = quads(_unpack_normal(n))
        ln = ns.norm(dim=-1, keepdim=True)
        pk = torch.where(ln > 0, _pack_normal(ns / ln.clamp(min=1e-300)), torch.zeros_like(ns[..., :2]))
        chain.append((quads(f), pk, quads(d) * 0.25))
    return chain


def _light_dir(light, u, v):
    M = _f64(light.inverse_view_projection).view(4, 4)
    x, y = u * 2 - 1, v * 2 - 1
    c = M[:, 0, None] * x + M[:, 1, None] * y + M[:, 3, None]
    return torch.nn.functional.normalize((c[:3] / c[3]).T - _f64(light.position), dim=1)


def _morton_xy(n):
    i = np.arange(n)
    x, y = np.zeros(n, np.int64), np.zeros(n, np.int64)
    for b in range(16):
        x |= ((i >> (2 * b)) & 1) << b
        y |= ((i >> (2 * b + 1)) & 1) << b
    return torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()


def _vpls(p, l, light):
    """VPLs in block order, and the cone source of every shadow block."""
    R = light.rsm_read_resolution
    chain = _rsm_level(p, l, light)
    lod = int(math.log2(light.rsm_render_resolution // R))
    f, n, d = chain[lod]
    x, y = _morton_xy(R * R)
    lp = _f64(light.position)
    dist = d[y, x, 0]
    pos = lp + _light_dir(light, (x + 0.5) / R, (y + 0.5) / R) * dist[:, None]
    out = {"flux": f[y, x], "normal": _unpack_normal(n[y, x]), "pos": pos, "area": dist ** 2 * light.val_area_factor}
    step = light.indirect_shadow_sample_interval
    xs, ys = x[::step], y[::step]
    u, v = (xs + light.indirect_shadow_sampling_offset) / R, (ys + light.indirect_shadow_sampling_offset) / R
    ds = chain[-1][2]
    rs = ds.shape[0]
    fx, fy = u * rs - 0.5, v * rs - 0.5
    x0, y0 = fx.floor().long(), fy.floor().long()
    ax, ay = (fx - x0)[:, None], (fy - y0)[:, None]
    at = lambda dy, dx: ds[(y0 + dy).clamp(0, rs - 1), (x0 + dx).clamp(0, rs - 1)]
    dd = (at(0, 0) * (1 - ax) + at(0, 1) * ax) * (1 - ay) + (at(1, 0) * (1 - ax) + at(1, 1) * ax) * ay
    out["cone"] = lp + _light_dir(light, u, v) * dd[:, :1]
    out["width"] = torch.clamp(2 * torch.sqrt((dd[:, 1] - dd[:, 0] ** 2).clamp(min=0)) / dd[:, 0],
                               min=light.indirect_shadow_super_val_width)
    out["interval"] = step
    return out


def _voxel_levels(hf):
    """Surface voxels of the boxes (binary32 decisions) and their exact means."""
    N, f = hf.workload.voxel_res, np.float32
    vm, vs = np.array(hf.volume.volume_world_min[:], f), f(hf.volume.voxel_size_in_world)
    grid = torch.zeros((N, N, N), dtype=torch.bool)
    for b in range(hf.scene.n_boxes):
        lo, hi = np.array(hf.boxes[b].min[:], f), np.array(hf.boxes[b].max[:], f)
        a, c = (lo - vm) / vs, (hi - vm) / vs
        first = np.maximum(0, np.ceil(a).astype(int) - 1)
        last = np.minimum(N - 1, np.floor(c).astype(int))
        for axis in range(3):
            for plane in (a[axis], c[axis]):
                if plane >= 0 and plane < N:
                    box = [slice(first[k], last[k] + 1) for k in range(3)]
                    box[axis] = slice(int(plane), int(plane) + 1)
                    grid[box[2], box[1], box[0]] = True
    levels = [grid.cuda().double()]
    while levels[-1].shape[0] > 1:
        levels.append(torch.nn.functional.avg_pool3d(levels[-1][None, None], 2)[0, 0])
    return levels


def _trilinear(tex, U, scale):
    n = tex.shape[0]
    u = (U * scale - 0.5).clamp(0, n - 1)
    i0 = u.floor().long()
    a, i1 = u - i0, (i0 + 1).clamp(max=n - 1)
    flat = tex.reshape(-1)
    r = 0.0
    for k in range(8):
        i = [(i1 if (k >> j) & 1 else i0)[:, j] for j in range(3)]
        w = 1.0
        for j in range(3):
            w = w * (a[:, j] if (k >> j) & 1 else 1 - a[:, j])
        r = r + flat[(i[2] * n + i[1]) * n + i[0]] * w
    return r


def _cone_visibility(hf, levels, cache, target, width):
    """Visibility of each (cache, target): the cone march through the voxel levels."""
    N, vs = hf.workload.voxel_res, float(hf.volume.voxel_size_in_world)
    t = target - cache
    ln = t.norm(dim=1)
    D = t / ln[:, None]
    U = (cache - _f64(hf.volume.volume_world_min)) / vs + 2 * D
    occ, vis = torch.zeros_like(ln), torch.empty_like(ln)
    step, dist, goal = torch.ones_like(ln), torch.zeros_like(ln), ln / vs - 2
    live = torch.arange(ln.numel(), device=ln.device)
    for _ in range(hf.config.max_cone_steps):
        U = U + D * step[:, None]
        dist = dist + step
        radius = dist * width
        lod = torch.log2(radius.clamp(min=1e-12)).clamp(0, len(levels) - 1)
        l0 = lod.floor().long()
        s = torch.zeros_like(dist)
        for l in range(len(levels)):
            w = torch.where(l0 == l, 1 - (lod - l0), torch.where(l0 + 1 == l, lod - l0, 0.0))
            at = w.nonzero()[:, 0]
            if at.numel():
                s[at] += _trilinear(levels[l], U[at], 2.0 ** -l) * w[at]
        occ = (1 - occ) * s + occ
        done = (dist >= goal) | (occ >= 1)
        vis[live] = (1 - occ).clamp(0, 1)
        keep = (~done).nonzero()[:, 0]
        if not keep.numel():
            break
        step = torch.clamp(radius * (2 / (1 - width)), min=1.0)
        live, U, D, occ, dist, step, goal, width = (q[keep] for q in (live, U, D, occ, dist, step, goal, width))
    return vis


def _pixels(p):
    """Cells of every pixel in the path's binary32 arithmetic, positions in 64 bits."""
    hf = p.hf
    w, h, f = hf.workload.width, hf.workload.height, torch.float32
    M = list(hf.frame.inverse_view_projection)
    d = p.depth
    ndc = lambda n: ((torch.arange(n, device="cuda", dtype=f) + 0.5) / torch.full((n,), float(n), device="cuda")) * 2.0 - 1.0
    nx, ny = ndc(w)[None, :], ndc(h)[:, None]
    row = lambda r, x, y, z: ((x * M[r]) + (y * M[r + 1]) + z * M[r + 2]) + M[r + 3]
    W = row(12, nx, ny, d)
    wp = [row(r, nx, ny, d) / W for r in (0, 4, 8)]
    x64 = ((torch.arange(w, device="cuda").double() + 0.5) / w * 2 - 1)[None, :]
    y64 = ((torch.arange(h, device="cuda").double() + 0.5) / h * 2 - 1)[:, None]
    W64 = row(12, x64, y64, d.double())
    wp64 = torch.stack([row(r, x64, y64, d.double()) / W64 for r in (0, 4, 8)], -1)
    nc = hf.config.n_cascades
    c = torch.full((h, w), nc - 1, dtype=torch.long, device="cuda")
    for k in reversed(range(nc - 1)):
        q = hf.volume.cascades[k]
        inside = torch.ones((h, w), dtype=torch.bool, device="cuda")
        for i in range(3):
            inside &= (wp[i] <= q.decision_max[i]) & (wp[i] >= q.decision_min[i])
        c = torch.where(inside, k, c)
    blend = torch.zeros((h, w), dtype=f, device="cuda")
    if hf.config.cascade_transition > 0:
        for k in range(nc - 1):
            q = hf.volume.cascades[k]
            m = torch.stack([q.decision_max[i] - wp[i] for i in range(3)] + [wp[i] - q.decision_min[i] for i in range(3)])
            zone = float(np.float32(q.world_voxel_size) * np.float32(hf.volume.cav_transition_zone_size))
            t = (1.0 - m.min(0).values / torch.full_like(d, zone)).clamp(0, 1)
            blend = torch.where(c == k, t, blend)
    return wp, wp64, c, blend


def _cells(hf, wp, c):
    """(x, y, z) / cell size of cascade c in binary32."""
    a = []
    for i in range(3):
        lo = torch.tensor([q.min[i] for q in hf.volume.cascades], device="cuda")[c]
        size = torch.tensor([q.world_voxel_size or 1.0 for q in hf.volume.cascades], device="cuda")[c]
        a.append((wp[i] - lo) / size)
    return a


def _allocated(p, wp, c, blend):
    """The atlas slots that the frame's pixels allocate: one per tile and cell,
    by the up / left comparison within 16 x 16 tiles (down / right for the
    transition cells)."""
    hf = p.hf
    res, nc, h, w = hf.config.cav_res, hf.config.n_cascades, *c.shape
    hp, wpad = (h + 15) // 16 * 16, (w + 15) // 16 * 16
    aw = nc * res
    taken = torch.zeros(res * res * aw, dtype=torch.bool, device="cuda")
    x, y = torch.arange(wpad, device="cuda")[None, :] % 16, torch.arange(hp, device="cuda")[:, None] % 16

    def key(cc, have):
        a = [q.nan_to_num(0.0).clamp(0, res - 1).long() for q in _cells(hf, wp, cc)]
        k = a[0] + a[1] * res + a[2] * res * res + cc * res ** 3
        full = torch.full((hp, wpad), -1, dtype=torch.long, device="cuda")
        full[:h, :w] = torch.where(have, k, -1)
        return full

    def shifted(k, dx, dy):  # the neighbour within the tile (itself at the tile's edge)
        j = torch.arange(wpad, device="cuda")
        i = torch.arange(hp, device="cuda")
        nj = (j // 16) * 16 + (j % 16 + dx).clamp(0, 15)
        ni = (i // 16) * 16 + (i % 16 + dy).clamp(0, 15)
        return k[ni][:, nj]

    def take(k, at):
        k = k[at & (k >= 0)].unique()
        cc = k // res ** 3
        b = k - cc * res ** 3
        bx, by, bz = b % res, b // res % res, b // (res * res)
        for o in range(8):
            ax, ly, lz = bx + (o & 1) + cc * res, by + (o >> 1 & 1), bz + (o >> 2)
            ok = (ax < aw) & (ly < res) & (lz < res)
            taken[((lz * res + ly) * aw + ax)[ok]] = True

    have = p.depth > 0.0001
    k1 = key(c, have)
    differs = (shifted(k1, 0, -1) != k1) & (shifted(k1, -1, 0) != k1) & (shifted(k1, -1, -1) != k1)
    take(k1, differs | ((x == 0) & (y == 0)))
    if hf.config.cascade_transition > 0:
        k2 = key((c + 1).clamp(max=nc - 1), have & (blend > 0) & (c < nc - 1))
        differs = (shifted(k2, 0, 1) != k2) & (shifted(k2, 1, 0) != k2) & (shifted(k2, 1, 1) != k2)
        take(k2, differs | ((x >= 14) & (y >= 14)))
    slots = taken.nonzero()[:, 0]
    ax = slots % aw
    cc = ax // res
    cell = torch.stack([ax - cc * res, slots // aw % res, slots // (aw * res)], 1).double()
    size = _f64(q.world_voxel_size for q in hf.volume.cascades)[cc]
    lo = torch.stack([_f64(q.min) for q in hf.volume.cascades])[cc]
    index = torch.full((taken.numel(),), slots.numel(), dtype=torch.long, device="cuda")
    index[slots] = torch.arange(slots.numel(), device="cuda")
    return cell * size[:, None] + lo, index


def _light(hf, vpls, pos):
    """SH coefficients [caches, 9, 3] of every cache."""
    ev = [1 / (2 * math.sqrt(PI)), math.sqrt(3) / (2 * math.sqrt(PI)), math.sqrt(15 / (4 * PI)),
          math.sqrt(5 / (16 * PI)), math.sqrt(15 / (16 * PI))]
    shadow = hf.config.indirect_shadow
    levels = _voxel_levels(hf) if shadow else None
    sh = torch.zeros((pos.shape[0], 9, 3), dtype=torch.float64, device="cuda")
    for v in vpls:
        lit = (v["flux"] > 0).any(1)
        for c0 in range(0, pos.shape[0], 1024):
            cache = pos[c0:c0 + 1024]
            t = v["pos"][None] - cache[:, None]
            d2 = (t * t).sum(-1)
            t = t / d2.sqrt()[..., None]
            g = (-(t * v["normal"][None]).sum(-1)).clamp(0, 1) / (d2 + v["area"])
            g = torch.where(lit[None], g, 0.0)
            if shadow:
                blocks = (g > 0).view(g.shape[0], -1, v["interval"]).any(-1)
                ci, bi = blocks.nonzero(as_tuple=True)
                vis = torch.zeros(blocks.shape, dtype=torch.float64, device="cuda")
                for k in range(0, ci.numel(), 1 << 20):
                    a, b = ci[k:k + (1 << 20)], bi[k:k + (1 << 20)]
                    vis[a, b] = _cone_visibility(hf, levels, cache[a], v["cone"][b], v["width"][b])
                g = g * vis.repeat_interleave(v["interval"], 1)
            x, y, z = t.unbind(-1)
            basis = [ev[0] * torch.ones_like(x), -ev[1] * y, ev[1] * z, -ev[1] * x, -ev[2] * x * y, ev[2] * y * z,
                     ev[3] * (3 * z * z - 1), ev[2] * x * z, ev[4] * (x * x - y * y)]
            for k in range(9 if hf.config.sh_order == 2 else 4):
                sh[c0:c0 + 1024, k] += (g * basis[k]) @ v["flux"]
    return sh


def _albedo(p):
    if p.albedo8 is None:
        return p.albedo.double()
    s = p.albedo8.double() / 255.0
    return torch.where(s <= 0.04045, s / 12.92, ((s + 0.055) / 1.055) ** 2.4)


def _normals(p):
    return _unpack_normal(p.normal16)


def _apply(p, wp, wp64, c, blend, sh, index):
    hf = p.hf
    res, nc = hf.config.cav_res, hf.config.n_cascades
    aw = nc * res
    n = _normals(p).reshape(-1, 3)
    x, y, z = n.unbind(1)
    q15 = -math.sqrt(15 * PI) / 8
    f0, f1 = math.sqrt(PI) / 2, math.sqrt(PI / 3)
    F = torch.stack([torch.full_like(x, f0), -f1 * y, f1 * z, -f1 * x, -q15 * x * y, q15 * y * z,
                     math.sqrt(5 * PI) / 16 * (3 * z * z - 1), q15 * x * z, math.sqrt(15 * PI) / 16 * (x * x - y * y)], 1)
    table = torch.cat([sh, torch.zeros_like(sh[:1])])  # the last: no cache there

    def irradiance(cc):
        a32 = torch.stack(_cells(hf, wp, cc), -1).reshape(-1, 3)
        cell = a32.clamp(-1e9, 1e9).trunc().nan_to_num(0.0)
        size = _f64(q.world_voxel_size or 1.0 for q in hf.volume.cascades)[cc].reshape(-1, 1)
        lo = torch.stack([_f64(q.min) for q in hf.volume.cascades])[cc].reshape(-1, 3)
        t = (wp64.reshape(-1, 3) - lo) / size - cell.double()
        base = cell.long()
        base[:, 0] += cc.reshape(-1) * res
        E = torch.zeros_like(n)
        for o in range(8):
            off = [o & 1, o >> 1 & 1, o >> 2]
            at = base + torch.tensor(off, device="cuda")
            ok = (at >= 0).all(1) & (at[:, 0] < aw) & (at[:, 1] < res) & (at[:, 2] < res)
            flat = ((at[:, 2] * res + at[:, 1]) * aw + at[:, 0]).clamp(0, index.numel() - 1)
            i = torch.where(ok, index[flat], table.shape[0] - 1)
            wgt = 1.0
            for j in range(3):
                wgt = wgt * (t[:, j] if off[j] else 1 - t[:, j])
            e = torch.zeros_like(n)
            for k in range(9 if hf.config.sh_order == 2 else 4):
                e += table[:, k][i] * F[:, k, None]
            E += e.clamp(min=0) * wgt[:, None]
        return E

    E = irradiance(c)
    if hf.config.cascade_transition > 0 and nc > 1:
        t = torch.where(c < nc - 1, blend, 0.0).double().reshape(-1, 1)
        E = torch.where(t > 0, E * (1 - t) + irradiance((c + 1).clamp(max=nc - 1)) * t, E)
    col = E.view(*c.shape, 3) * _albedo(p) / PI
    col = torch.where((p.depth >= 0.00001)[..., None], col, 0.0)
    if hf.config.output_format == abi.OUTPUT_RGBA16F:
        col = torch.cat([col, torch.ones_like(col[..., :1])], -1)
    return col


def _brute(p, vpls, materials):
    """Unshadowed sum over every VPL; materials: normalised Blinn-Phong with metallic."""
    hf = p.hf
    _, wp64, _, _ = _pixels(p)
    pos, n, base = wp64.reshape(-1, 3), _normals(p).reshape(-1, 3), _albedo(p).reshape(-1, 3)
    out = torch.zeros_like(pos)
    cam = _f64(hf.frame.camera_position)
    for k in range(0, pos.shape[0], 16384):
        P, Nn, B = pos[k:k + 16384], n[k:k + 16384], base[k:k + 16384]
        for v in vpls:
            t = v["pos"][None] - P[:, None]
            d2 = (t * t).sum(-1)
            t = t / d2.sqrt()[..., None]
            cos = (t @ Nn[..., None])[..., 0].clamp(0, 1)
            g = (-(t * v["normal"][None]).sum(-1)).clamp(0, 1) * cos / (d2 + v["area"])
            if materials is None:
                out[k:k + 16384] += (g @ v["flux"]) * B / PI
                continue
            r, m = (materials.reshape(-1, 2)[k:k + 16384, q].double()[:, None] for q in (0, 1))
            e = 2 / (r ** 4 + 0.0005)
            to_cam = torch.nn.functional.normalize(cam - P, dim=1)
            hv = torch.nn.functional.normalize(to_cam[:, None] + t, dim=-1)
            bp = (e + 8) / (8 * PI) * (hv @ Nn[..., None])[..., 0].clamp(0, 1) ** e
            diffuse, spec = B * (1 - m) + 0.02 * m, 0.04 * (1 - m) + B * m
            out[k:k + 16384] += (g @ v["flux"]) * diffuse / PI + ((g * bp) @ v["flux"]) * spec
    return torch.where((p.depth.reshape(-1, 1) >= 0.00001), out, 0.0).view(*p.depth.shape, 3)


def _cast(hf, origin, d):
    """Nearest box surface along each ray: (distance, box, axis)."""
    best = torch.full((d.shape[0],), math.inf, dtype=torch.float64, device="cuda")
    box, axis = torch.full_like(best, -1, dtype=torch.long), torch.zeros_like(best, dtype=torch.long)
    for b in range(hf.scene.n_boxes):
        q = hf.boxes[b]
        t0, t1 = (_f64(q.min) - origin) / d, (_f64(q.max) - origin) / d
        near, na = torch.minimum(t0, t1).max(1)
        far, fa = torch.maximum(t0, t1).min(1)
        t, a = (far, fa) if q.inward else (near, na)
        hit = (near <= far) & (t > 1e-6) & (t < best)
        best, box, axis = torch.where(hit, t, best), torch.where(hit, b, box), torch.where(hit, a, axis)
    return best, box, axis


def _exact_mesh(p, case):
    hf = p.hf
    cam, w, h = hf.camera, case["width"], case["height"]
    fwd = torch.nn.functional.normalize(_f64(cam.direction), dim=0)
    up = _f64(cam.up)
    right = torch.nn.functional.normalize(torch.linalg.cross(up, fwd), dim=0)
    up = torch.linalg.cross(fwd, right)
    ty = math.tan(math.radians(cam.fov_y_deg) * 0.5)
    x = (torch.arange(w, device="cuda").double() + 0.5) / w * 2 - 1
    y = (torch.arange(h, device="cuda").double() + 0.5) / h * 2 - 1
    d = (fwd + right * (ty * cam.aspect) * x[None, :, None] + up * ty * y[:, None, None]).reshape(-1, 3)
    d = torch.nn.functional.normalize(d, dim=1)
    albedos = torch.stack([_f64(hf.boxes[b].albedo) for b in range(hf.scene.n_boxes)])

    def normal(axis, dirs):
        s = torch.gather(dirs, 1, axis[:, None])
        return torch.zeros_like(dirs).scatter_(1, axis[:, None], -torch.sign(s))

    t, box, axis = _cast(hf, _f64(cam.position), d)
    point = _f64(cam.position) + d * t[:, None]
    M = _f64(hf.frame.view_projection).view(4, 4)
    clip = point @ M[2:, :3].T + M[2:, 3]
    out = {"depth": (clip[:, 0] / clip[:, 1]).view(h, w), "normal16": None, "normal": normal(axis, d).view(h, w, 3),
           "albedo": albedos[box].view(h, w, 3), "flux": [], "rsm_normal": None, "depth_lin_sq": [],
           "voxels": None, "mips": None}
    for l in range(case["lights"]):
        L, R = hf.lights[l], hf.lights[l].rsm_render_resolution
        u = ((torch.arange(R, device="cuda").double() + 0.5) / R)
        d = _light_dir(L, u.repeat(R), u.repeat_interleave(R))
        t, box, axis = _cast(hf, _f64(L.position), d)
        cos = (d @ _f64(L.direction)).clamp(0, 1)
        falloff = (cos - L.cos_half_angle).clamp(0, 1) / (1 - L.cos_half_angle)
        k = falloff * 2 * PI * (1 - L.cos_half_angle) * cos / R / R / PI
        out["flux"].append((albedos[box] * _f64(L.intensity) * k[:, None]).view(R, R, 3))
        out["depth_lin_sq"].append(torch.stack([t, t * t], 1).view(R, R, 2))
    return out


def _exact_train(case, seed):
    X, Y, params, m, v = (t.double() for t in _train_data(case, seed))
    n = X.shape[0]
    P = params.clone().requires_grad_(True)
    mats, o = [], 0
    for rows, cols in ((64, 32), (64, 64), (64, 64), (2, 64)):
        mats.append((P[o:o + rows * cols].view(rows, cols), P[o + rows * cols:o + rows * cols + rows]))
        o += rows * cols + rows
    a = X
    for k, (W, b) in enumerate(mats):
        z = a @ W.T + b
        a = z * torch.sigmoid(1.702 * z) if k < 3 else z
    vis, conf = torch.sigmoid(a[:, 0]), torch.sigmoid(a[:, 1])
    target = ((vis - Y).abs() < 0.03).double().detach()
    bce = lambda q, t: torch.nn.functional.binary_cross_entropy(q, t, reduction="sum")
    losses = torch.stack([bce(vis, Y), bce(conf, target)])
    (losses.sum() / n).backward()
    g, step = P.grad, 501
    m = 0.9 * m + 0.1 * g
    v = 0.999 * v + 0.001 * g * g
    update = (m / (1 - 0.9 ** step)) / ((v / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return {"params": params - 1e-3 * (update + 1e-4 * params), "m": m, "v": v, "loss": losses.detach()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    # The surrogate's thresholded decisions and the R11F_G11F_B10F envmaps
    # have no 64-bit value that the outputs should be near.
    if kind == "batch" or case.get("surrogate") or case.get("specular"):
        return None
    p = _pipeline(case, seed)
    if kind == "mesh":
        return _exact_mesh(p, case)
    _fill_inputs(p, seed)
    hf = p.hf
    vpls = [_vpls(p, l, hf.lights[l]) for l in range(case["lights"])]
    if kind == "brute":
        return _brute(p, vpls, p.rough_metal.float() / 255.0 if case["materials"] else None)
    wp, wp64, c, blend = _pixels(p)
    pos, index = _allocated(p, wp, c, blend)
    sh = _light(hf, vpls, pos)
    return {"radiance": _apply(p, wp, wp64, c, blend, sh, index), "counter": None}
