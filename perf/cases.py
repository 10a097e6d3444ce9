"""The framework's work as its users call it, one case per kind of call and size.

Kinds (each through the public Python entry points):

``render``   ``GpuScene.render``: progressive frames, previews and many-sample
             frames of the procedural scenes (Cornell box, seven materials,
             icosphere field, hair), both random streams, with and without
             AOVs.
``batch``    ``render_batch``: many scenes of uneven size and resolution in one
             launch per bounce.
``dynamic``  one frame of an animation: new vertex positions on the device,
             the acceleration structure refit or rebuilt, one frame rendered.
``trace``    ``GpuScene.trace``: closest-hit and any-hit queries of one ray set.
``denoise``  ``Denoiser.denoise``: a rendered frame through the learned
             denoiser (one network pass, or the mirror ensemble).
``train``    ``Denoiser.train_step``: one Adam step on a batch of crops; the
             loss and the updated weights come back.

Renders have no closed-form value (a path's discrete choices follow the
rounding of every step), so ``exact`` covers the ray queries, the denoiser and
the training step.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

from pupiloptixlab_gb300 import abi, scenes
from pupiloptixlab_gb300.api import Context, GpuScene, render_batch
from pupiloptixlab_gb300.denoiser import Denoiser

_CTX = None


def _ctx() -> Context:
    """One context per process, as a program holds it."""
    global _CTX
    if _CTX is None:
        _CTX = Context(torch.cuda.current_device())
    return _CTX


# ------------------------------------------------------------------ the cases

def listed() -> list:
    return [
        # the smallest render: one progressive frame of a viewer (the reference's stream), AOVs on
        {"name": "preview_cornell_256", "kind": "render", "scene": "cornell", "width": 256, "height": 256, "spp": 1,
         "depth": 4, "rng": abi.RNG_REF_LCG, "size": 0, "aovs": True},
        # the plain small configuration: Cornell box, 256 x 256, 16 spp, depth 4
        {"name": "cornell_256_16spp", "kind": "render", "scene": "cornell", "width": 256, "height": 256, "spp": 16,
         "depth": 4, "rng": abi.RNG_PCG32, "size": 0, "aovs": False},
        # all seven materials and a checkerboard, odd film size, a few samples
        {"name": "materials_613x347_5spp", "kind": "render", "scene": "spheres", "width": 613, "height": 347, "spp": 5,
         "depth": 6, "rng": abi.RNG_PCG32, "size": 0, "aovs": True},
        # curves: 10 k cubic strands, odd film size
        {"name": "hair_641x361_8spp", "kind": "render", "scene": "hair", "width": 641, "height": 361, "spp": 8,
         "depth": 8, "rng": abi.RNG_PCG32, "size": 10000, "aovs": False},
        # one progressive 1080p frame of the 1M-triangle field (what a viewer shows, and a denoiser's input)
        {"name": "field_1080p_1spp", "kind": "render", "scene": "field", "width": 1920, "height": 1080, "spp": 1,
         "depth": 8, "rng": abi.RNG_REF_LCG, "size": 200, "aovs": True},
        # the headline: 1M triangles, 1080p, 64 spp, depth 8
        {"name": "field_1080p_64spp", "kind": "render", "scene": "field", "width": 1920, "height": 1080, "spp": 64,
         "depth": 8, "rng": abi.RNG_PCG32, "size": 200, "aovs": True},
        # scenes of uneven size and resolution in one launch per bounce
        {"name": "batch_12_scenes_4spp", "kind": "batch", "scenes": 12, "largest": 200, "spp": 4, "depth": 8},
        # animation, 4.1M triangles: refit and one sample per pixel
        {"name": "dynamic_refit_4m", "kind": "dynamic", "how": "refit", "size": 800, "width": 1280, "height": 720,
         "depth": 6, "spp": 1},
        # the same with a full-quality rebuild each frame
        {"name": "dynamic_rebuild_4m", "kind": "dynamic", "how": "rebuild", "size": 800, "width": 1280, "height": 720,
         "depth": 6, "spp": 1},
        # incoherent ray queries, closest and any hit
        {"name": "trace_1m_rays", "kind": "trace", "size": 40, "rays": 1 << 20},
        # one rendered 1080p frame through the network
        {"name": "denoise_1080p", "kind": "denoise", "width": 1920, "height": 1080, "ensemble": False},
        # the stated training step: 16 crops of 256 x 256
        {"name": "train_16x256", "kind": "train", "batch": 16, "crop": 256},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["render", "render", "render", "batch", "dynamic", "trace", "denoise", "train"])
    if kind == "render":
        scene = rng.choice(["cornell", "spheres", "hair", "field"])
        size = {"hair": _log_int(rng, 300, 20000), "field": _log_int(rng, 8, 200)}.get(scene, 0)
        return {"kind": kind, "scene": scene, "width": _log_int(rng, 96, 1920), "height": _log_int(rng, 64, 1080),
                "spp": _log_int(rng, 1, 32), "depth": rng.randint(3, 8),
                "rng": rng.choice([abi.RNG_REF_LCG, abi.RNG_PCG32]), "size": size, "aovs": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "scenes": _log_int(rng, 2, 16), "largest": _log_int(rng, 8, 200),
                "spp": _log_int(rng, 1, 8), "depth": rng.randint(4, 8)}
    if kind == "dynamic":
        return {"kind": kind, "how": rng.choice(["refit", "rebuild", "fast"]), "size": _log_int(rng, 4, 800),
                "width": _log_int(rng, 160, 1280), "height": _log_int(rng, 90, 720), "depth": rng.randint(3, 6),
                "spp": rng.randint(1, 2)}
    if kind == "trace":
        return {"kind": kind, "size": _log_int(rng, 1, 200), "rays": _log_int(rng, 256, 1 << 21)}
    if kind == "denoise":
        return {"kind": kind, "width": _log_int(rng, 64, 1920), "height": _log_int(rng, 64, 1080),
                "ensemble": rng.random() < 0.4}
    return {"kind": kind, "batch": rng.randint(1, 16), "crop": 16 * rng.randint(2, 16)}


# ------------------------------------------------------------------ inputs

def _scene(which: str, size: int, width: int, height: int, depth: int, seed: int):
    r = np.random.default_rng(seed)
    if which == "field":  # the icosphere field; its meshes are shared by the instances
        return scenes.pooled_field(seed, size, width, height, depth, pool=scenes.mesh_pool(min(size, 16), seed=seed % 1009))
    if which == "cornell":
        sc = scenes.cornell_box(width, height, depth)
        eye, target, fov = (0.0, 1.0, 3.8), (0.0, 1.0, 0.0), 40.0
    elif which == "spheres":
        sc = scenes.material_spheres(width, height, depth)
        eye, target, fov = (0.0, 3.0, 12.0), (0.0, 1.0, 0.0), 35.0
    else:
        sc = scenes.hair_scene(width, height, num_strands=size, points=16, radius=0.006, max_depth=depth, seed=seed)
        eye, target, fov = (0.0, 2.2, 5.5), (0.0, 1.3, 0.0), 35.0
    eye = tuple(e + float(d) for e, d in zip(eye, r.uniform(-0.2, 0.2, 3)))
    sc.camera = scenes.camera(fov, width / height, scenes.look_at_to_world(eye, target))
    return sc


def _object_positions(sc) -> torch.Tensor:
    return torch.from_numpy(np.concatenate([m.positions for m in sc.meshes])).cuda()


def _rays(sc, size: int, count: int, seed: int) -> torch.Tensor:
    """Half the rays leave the camera's side of the field towards it, half start inside it."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    half = 10.0 * (size / 200.0) ** (1.0 / 3.0)
    d = torch.randn(count, 3, generator=g, device="cuda")
    o = torch.rand(count, 3, generator=g, device="cuda") * (2 * half) - half
    o[:, 1] += half + 1.5
    out = torch.arange(count, device="cuda") % 2 == 0
    aim = o - torch.tensor([0.0, 1.4 * half, 3.8 * half + 2.0], device="cuda")
    d = torch.where(out[:, None], aim, d)
    o = torch.where(out[:, None], o - aim, o)
    d = d / d.norm(dim=1, keepdim=True)
    rays = torch.empty(count, 8, device="cuda")
    rays[:, 0:3], rays[:, 3], rays[:, 4:7], rays[:, 7] = o, 0.001, d, 1e16
    return rays


def _smooth(g, channels: int, height: int, width: int) -> torch.Tensor:
    """Piecewise smooth random image (height, width, channels) in [0, 1]."""
    low = torch.rand(1, channels, max(2, height // 24), max(2, width // 24), generator=g, device="cuda")
    return F.interpolate(low, size=(height, width), mode="bilinear", align_corners=False)[0].permute(1, 2, 0)


def _frame(seed: int, height: int, width: int, spp: float) -> tuple:
    """A path tracer's frame in form: noisy HDR colour, its clean colour, albedo, unit normals."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    albedo = 0.1 + 0.8 * _smooth(g, 3, height, width)
    clean = albedo * (0.05 + 3.0 * _smooth(g, 1, height, width) ** 2)
    noise = torch.empty(height, width, 1, device="cuda").exponential_(1.0, generator=g) - 1.0
    noisy = (clean * (1.0 + noise / math.sqrt(spp))).clamp_(min=0.0)
    normal = _smooth(g, 3, height, width) * 2.0 - 1.0
    normal = normal / normal.norm(dim=-1, keepdim=True).clamp_(min=1e-3)
    return noisy, clean, albedo, normal


def _network(seed: int, lr: float = 1e-3) -> tuple:
    """A denoiser whose weights are past their start (the output layer starts at zero), and those weights."""
    dn = Denoiser(_ctx(), lr=lr, seed=seed + 1)
    p = dn.get_params()
    r = np.random.default_rng(seed)
    cin, cout, off = dn.layers[-1]
    w = np.zeros((cout, 9, cin), np.float32)
    w[:3] = r.normal(0.0, 0.01, (3, 9, cin))
    p[off:off + w.size] = w.ravel()
    for cin, cout, off in dn.layers[:-1]:
        b = off + 9 * cin * cout
        p[b:b + cout] = r.normal(0.0, 0.02, cout)
    dn.set_params(p)
    return dn, p


def _train_inputs(case: dict, seed: int) -> tuple:
    n, c = case["batch"], case["crop"]
    frames = [_frame(seed * 64 + k, c, c, float(2 ** (k % 8))) for k in range(n)]
    inputs = torch.stack([torch.cat([f[0], f[2], f[3]], dim=-1) for f in frames]).to(torch.float16)
    return inputs.contiguous(), torch.stack([f[1] for f in frames]).contiguous()


def _adam_state(dn) -> np.ndarray:
    """Moments of a run under way: 1000 steps done, second moments of the gradients' usual size."""
    n = dn.num_params
    st = np.zeros(2 * n + 4, np.float32)
    st[n:2 * n] = 1e-6
    st[2 * n] = 1000.0
    st[2 * n + 3] = 1e-3
    return st


def _batch_layout(case: dict) -> list:
    """(instances, width, height) of every scene of a batch: log-uniform instance counts, the film sizes in turn."""
    r = np.random.default_rng([case["scenes"], case["largest"]])
    sizes = [(256, 256), (512, 512), (640, 360), (333, 251)]
    return [(int(round(math.exp(r.uniform(math.log(2), math.log(case["largest"]))))), *sizes[k % 4])
            for k in range(case["scenes"])]


def _batch_scenes(case: dict, seed: int) -> list:
    pool = scenes.mesh_pool(12, seed=seed % 1009)
    return [scenes.pooled_field(1000 * seed + k, count, w, h, case["depth"], pool=pool)
            for k, (count, w, h) in enumerate(_batch_layout(case))]


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "render":
        sc = _scene(case["scene"], case["size"], case["width"], case["height"], case["depth"], seed)
        g = GpuScene(_ctx(), sc)
        return {"case": case, "scene": g, "buffers": g.alloc_buffers(aovs=case["aovs"]), "seed": (seed * 4096) & 0x7FFFFFFF}
    if kind == "batch":
        gs = [GpuScene(_ctx(), sc) for sc in _batch_scenes(case, seed)]
        return {"case": case, "scenes": gs, "buffers": [g.alloc_buffers(aovs=False) for g in gs], "seed": (seed * 4096) & 0x7FFFFFFF}
    if kind == "dynamic":
        sc = _scene("field", case["size"], case["width"], case["height"], case["depth"], seed)
        g = GpuScene(_ctx(), sc, bvh_flags=abi.BVH_FAST_BUILD if case["how"] == "fast" else 0)
        pos = _object_positions(sc)
        gen = torch.Generator(device="cuda").manual_seed(seed)
        pos = pos + 0.002 * torch.randn(pos.shape, generator=gen, device="cuda")
        return {"case": case, "scene": g, "positions": pos, "buffers": g.alloc_buffers(aovs=False), "seed": (seed * 4096) & 0x7FFFFFFF}
    if kind == "trace":
        sc = _scene("field", case["size"], 64, 64, 4, seed)
        return {"case": case, "scene": GpuScene(_ctx(), sc), "rays": _rays(sc, case["size"], case["rays"], seed)}
    if kind == "denoise":
        w, h = case["width"], case["height"]
        noisy, _, albedo, normal = _frame(seed, h, w, 32.0)
        color = torch.cat([noisy, torch.ones(h, w, 1, device="cuda")], dim=-1)
        buffers = {"accum": color.reshape(-1, 4).contiguous(), "albedo": albedo.reshape(-1, 3).contiguous(),
                   "normal": normal.reshape(-1, 3).contiguous()}
        return {"case": case, "denoiser": _network(seed)[0], "buffers": buffers}
    dn, _ = _network(seed)
    dn.set_state(_adam_state(dn))
    inputs, targets = _train_inputs(case, seed)
    return {"case": case, "denoiser": dn, "inputs": inputs, "targets": targets}


# ------------------------------------------------------------------ one pass

def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "render":
        return state["scene"].render(case["spp"], seed=state["seed"], rng=case["rng"], buffers=state["buffers"])
    if kind == "batch":
        return render_batch(_ctx(), state["scenes"], case["spp"], seed=state["seed"], buffers=state["buffers"])
    if kind == "dynamic":
        g = state["scene"]
        g.update_all_vertices(state["positions"])
        if case["how"] == "refit":
            g.refit()
        else:
            g.build_bvh()
        return g.render(case["spp"], seed=state["seed"], buffers=state["buffers"])
    if kind == "trace":
        closest = state["scene"].trace(state["rays"])
        occluded = state["scene"].trace(state["rays"], anyhit=True)
        return {"t": closest[:, 0], "prim": closest.view(torch.int32)[:, 1], "u": closest[:, 2], "v": closest[:, 3],
                "occluded": occluded[:, 0]}
    if kind == "denoise":
        out, stats, _ = state["denoiser"].denoise(state["buffers"], case["width"], case["height"],
                                                  ensemble=case["ensemble"])
        return {"output": out, "fallback_tiles": stats.fallback_tiles}
    dn = state["denoiser"]
    dn.train_step(state["inputs"], state["targets"])
    return {"loss": dn.read_loss(), "params": dn.get_params()}


# ------------------------------------------------------------------ necessary work

# Per ray: 16 four-wide nodes (4 boxes of 6 fused multiply-adds and 11 comparisons), 3 triangle tests.
_RAY_FLOPS = 16 * 4 * 23 + 3 * 60
_SHADE_FLOPS = 300
# Closest-hit and shadow rays of one path, by scene (open scenes lose paths to the environment).
_RAYS = {"cornell": 6.0, "spheres": 3.0, "hair": 3.5, "field": 2.7}
_TRI_BYTES = 36 + 24  # vertex positions, shared normals and indices


def _triangles(scene: str, size: int) -> int:
    return {"cornell": 36, "spheres": 9100, "hair": size * 13 * 4, "field": 5120 * size + 8192}[scene]


def _conv_flops(pixels: float) -> float:
    """Multiply-adds of the 14 convolutions of the network, times two."""
    spec = [(16, 32, 1), (32, 32, 1), (32, 48, 4), (48, 48, 4), (48, 64, 16), (64, 64, 16), (64, 128, 64),
            (128, 128, 64), (128, 256, 256), (384, 128, 64), (192, 64, 16), (112, 48, 4), (80, 32, 1), (32, 3, 1)]
    return sum(2.0 * 9 * ci * co * pixels / div for ci, co, div in spec)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("render", "dynamic"):
        scene = case.get("scene", "field")
        tris = _triangles(scene, case["size"])
        px = case["width"] * case["height"]
        buffers = 32 + (28 if case.get("aovs") else 0)
        flops = px * case["spp"] * _RAYS[scene] * (_RAY_FLOPS + _SHADE_FLOPS)
        # an animated frame also writes every triangle's record and the nodes over it
        extra = tris * (48 + 128 / 2.5) if kind == "dynamic" else 0
        return {"bytes": float(tris * _TRI_BYTES + px * buffers + extra), "flops": float(flops)}
    if kind == "batch":
        layout = _batch_layout(case)
        px = sum(w * h for _, w, h in layout)
        tris = sum(_triangles("field", count) for count, _, _ in layout)
        return {"bytes": float(tris * _TRI_BYTES + 32 * px),
                "flops": float(px * case["spp"] * _RAYS["field"] * (_RAY_FLOPS + _SHADE_FLOPS))}
    if kind == "trace":
        return {"bytes": float(_triangles("field", case["size"]) * 36 + case["rays"] * (32 + 16 + 16)),
                "flops": float(2 * case["rays"] * _RAY_FLOPS)}
    if kind == "denoise":
        px = case["width"] * case["height"]
        passes = 2 if case["ensemble"] else 1
        return {"bytes": float(px * (16 + 12 + 12 + 16) + 2 * 1259072), "flops": float(passes * _conv_flops(px))}
    px = case["batch"] * case["crop"] ** 2
    # forward, data gradient (not of the first layer) and weight gradient; weights and both moments read and written
    flops = 3.0 * _conv_flops(px) - 2.0 * 9 * 16 * 32 * px
    return {"bytes": float(px * (18 + 12) + 1259072 * 4 * 6), "flops": flops}


# ------------------------------------------------------------------ values in 64 bits

def _exact_trace(case: dict, seed: int):
    sc = _scene("field", case["size"], 64, 64, 4, seed)
    rays = _rays(sc, case["size"], case["rays"], seed).double()
    tris, spheres = [], []
    for inst in sc.instances:
        m = torch.from_numpy(np.asarray(inst["to_world"], np.float32).astype(np.float64)).cuda()
        if inst["shape_type"] == abi.SHAPE_MESH:
            mesh = sc.meshes[inst["shape_index"]]
            p = torch.from_numpy(mesh.positions.astype(np.float64)).cuda() @ m[:3, :3].T + m[:3, 3]
            tris.append(p[torch.from_numpy(mesh.indices.astype(np.int64)).cuda()])
        else:
            c, r = sc.spheres[inst["shape_index"]]
            center = m[:3, :3] @ torch.tensor(c, dtype=torch.float64, device="cuda") + m[:3, 3]
            spheres.append((center, r * float(m[:3, 0].norm())))
    tris = torch.cat(tris)
    if tris.shape[0] * rays.shape[0] > 2e10:
        return None
    n = rays.shape[0]
    best = torch.full((n,), 1e16, dtype=torch.float64, device="cuda")
    u = torch.zeros(n, dtype=torch.float64, device="cuda")
    v = torch.zeros_like(u)
    prim = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    step_r = 4096
    step_t = 8192
    for a in range(0, n, step_r):
        o, d = rays[a:a + step_r, None, 0:3], rays[a:a + step_r, None, 4:7]
        for b in range(0, tris.shape[0], step_t):
            t = tris[b:b + step_t]
            p0, e1, e2 = t[None, :, 0], (t[:, 1] - t[:, 0])[None], (t[:, 2] - t[:, 0])[None]
            q = torch.linalg.cross(d.expand(-1, t.shape[0], -1), e2.expand(d.shape[0], -1, -1))
            det = (e1 * q).sum(-1)
            s = o - p0
            uu = (s * q).sum(-1) / det
            rr = torch.linalg.cross(s, e1.expand_as(s))
            vv = (d * rr).sum(-1) / det
            tt = (e2 * rr).sum(-1) / det
            ok = (uu >= 0) & (vv >= 0) & (uu + vv <= 1) & (tt > 0.001)
            tt = torch.where(ok, tt, torch.full_like(tt, 1e17))
            m, at = tt.min(dim=1)
            better = m < best[a:a + step_r]
            rows = torch.arange(m.shape[0], device="cuda")
            best[a:a + step_r] = torch.where(better, m, best[a:a + step_r])
            prim[a:a + step_r] = torch.where(better, at + b, prim[a:a + step_r])
            u[a:a + step_r] = torch.where(better, uu[rows, at], u[a:a + step_r])
            v[a:a + step_r] = torch.where(better, vv[rows, at], v[a:a + step_r])
    o, d = rays[:, 0:3], rays[:, 4:7]
    for k, (c, r) in enumerate(spheres):
        f = o - c
        aa, bb, cc = (d * d).sum(-1), (f * d).sum(-1), (f * f).sum(-1) - r * r
        disc = bb * bb - aa * cc
        root = disc.clamp(min=0).sqrt()
        for sign in (-1.0, 1.0):
            t = (-bb + sign * root) / aa
            better = (disc >= 0) & (t > 0.001) & (t < best)
            best = torch.where(better, t, best)
            prim = torch.where(better, torch.full_like(prim, tris.shape[0] + k), prim)
            u, v = torch.where(better, torch.zeros_like(u), u), torch.where(better, torch.zeros_like(v), v)
    return {"t": best, "prim": prim, "u": u, "v": v, "occluded": (prim >= 0).double()}


def _net64(p: np.ndarray, layers: list, rgbfeat: torch.Tensor) -> tuple:
    """The network in 64 bits on (n, h, w, 9): (log-domain prediction (n, 3, h, w), its parameters)."""
    x = rgbfeat.double()
    x0 = torch.cat([torch.log1p(x[..., :3].clamp(min=0.0)), x[..., 3:9], torch.zeros(*x.shape[:3], 7, device=x.device,
                                                                                    dtype=torch.float64)], dim=-1)
    x0 = x0.permute(0, 3, 1, 2)
    params = []
    for cin, cout, off in layers:
        nw = 9 * cin * cout
        w = torch.from_numpy(p[off:off + nw].astype(np.float64).reshape(cout, 3, 3, cin)).cuda().permute(0, 3, 1, 2)
        params.append((w.contiguous().requires_grad_(True),
                       torch.from_numpy(p[off + nw:off + nw + cout].astype(np.float64)).cuda().requires_grad_(True)))

    def conv(i, a):
        a = F.conv2d(a, params[i][0], params[i][1], padding=1)
        return a if i == 13 else torch.relu(a)

    def up(a):
        return F.interpolate(a, scale_factor=2, mode="nearest")

    e0 = conv(1, conv(0, x0))
    e1 = conv(3, conv(2, F.avg_pool2d(e0, 2)))
    e2 = conv(5, conv(4, F.avg_pool2d(e1, 2)))
    e3 = conv(7, conv(6, F.avg_pool2d(e2, 2)))
    b4 = conv(8, F.avg_pool2d(e3, 2))
    d3 = conv(9, torch.cat([up(b4), e3], dim=1))
    d2 = conv(10, torch.cat([up(d3), e2], dim=1))
    d1 = conv(11, torch.cat([up(d2), e1], dim=1))
    d0 = conv(12, torch.cat([up(d1), e0], dim=1))
    return conv(13, d0)[:, :3] + x0[:, :3], params


def _exact_denoise(case: dict, seed: int):
    w, h = case["width"], case["height"]
    dn, p = _network(seed)
    noisy, _, albedo, normal = _frame(seed, h, w, 32.0)
    pad = (0, 0, 0, -w % 16, 0, -h % 16)
    x = F.pad(torch.cat([noisy, albedo, normal], dim=-1), pad)[None]
    with torch.no_grad():
        log = _net64(p, dn.layers, x)[0]
        if case["ensemble"]:
            log = 0.5 * (log + _net64(p, dn.layers, x.flip(2))[0].flip(3))
        rgb = torch.expm1(log)[0].clamp(min=0.0).permute(1, 2, 0)[:h, :w]
        # a tile whose mean luminance moves by more than max(25 %, 4 standard errors) keeps its raw colour
        lum = torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64, device="cuda")
        raw = noisy.double()
        th, tw = (h + 15) // 16, (w + 15) // 16

        def tiles(a):
            return F.pad(a, (0, -w % 16, 0, -h % 16)).reshape(th, 16, tw, 16).sum(dim=(1, 3))

        count = tiles(torch.ones(h, w, dtype=torch.float64, device="cuda"))
        lr, ld = raw @ lum, rgb @ lum
        mean, mden = tiles(lr) / count, tiles(ld) / count
        se = ((tiles(lr * lr) / count - mean * mean).clamp(min=0.0) / count).sqrt()
        keep = (mden - mean).abs() > torch.maximum(0.25 * mean, 4.0 * se)
        mask = keep.repeat_interleave(16, 0).repeat_interleave(16, 1)[:h, :w, None]
        out = torch.cat([torch.where(mask, raw, rgb), torch.ones(h, w, 1, dtype=torch.float64, device="cuda")], dim=-1)
    return {"output": out.reshape(-1, 4), "fallback_tiles": None}


def _exact_train(case: dict, seed: int):
    dn, p = _network(seed)
    st = _adam_state(dn).astype(np.float64)
    inputs, targets = _train_inputs(case, seed)
    log, params = _net64(p, dn.layers, inputs)
    loss = (log - torch.log1p(targets.double().clamp(min=0.0)).permute(0, 3, 1, 2)).abs().mean()
    loss.backward()
    grad = torch.cat([torch.cat([w.grad.permute(0, 2, 3, 1).reshape(-1), b.grad]) for w, b in params]).cpu().numpy()
    n = dn.num_params
    t = st[2 * n] + 1.0
    m = 0.9 * st[:n] + 0.1 * grad
    v = 0.999 * st[n:2 * n] + 0.001 * grad * grad
    new = p.astype(np.float64) - st[2 * n + 3] * (m / (1 - 0.9 ** t)) / (np.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    return {"loss": loss.detach().item(), "params": new}


def exact(case: dict, seed: int):
    if case["kind"] == "trace":
        return _exact_trace(case, seed)
    if case["kind"] == "denoise":
        return _exact_denoise(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return None
