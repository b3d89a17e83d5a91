"""Performance cases: the work that users of this framework have it do, through its public
Python entry points, over the range of sizes that they use.

Kinds of case:

* ``trace``: ray queries against a tree that the program keeps (closest or any hit, exact or
  fast mode, device or host buffers).
* ``export``: a tiny tree built and read back node by node (parity checks, tools).
* ``frame``: a tree rebuilt from new geometry and queried at once (animated scenes, a served
  job that brings its own scene).
* ``batch``: many scenes' trees from one batched build, each queried.
* ``render``: a whole path-traced film of a loaded scene.
* ``mlp``: the learned directional proposal's forward pass and its training gradients.

Geometry: ``soup`` (triangles of log-uniform size spread over the unit cube), ``room`` (the
34-triangle room with its 2-triangle light) and ``spheres`` (tessellated spheres of assorted
materials in a room).  Rays: ``random`` (origins and directions uniform), ``shadow`` (towards
a point of the scene, bounded by its distance) and ``camera`` (a jittered pinhole grid).
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

import cavalry_b200 as cav
from cavalry_b200 import scenes

_MODES = {"exact": cav.TRACE_EXACT, "fast": cav.TRACE_FAST}
_CONTEXT = []


def _ctx() -> cav.Context:
    """One context for the process, as a program keeps it."""
    if not _CONTEXT:
        _CONTEXT.append(cav.Context(0))
    return _CONTEXT[0]


# ------------------------------------------------------------------------------- cases
def listed() -> list[dict]:
    return [
        # A picking or probe query on the smallest scene: launch latency.
        {"name": "query_room", "kind": "trace", "scene": "room", "tris": 36, "rounds": 2, "rays": "random",
         "n": 4096, "mode": "exact", "buffers": "device"},
        # The closest-hit benchmark: incoherent rays over a dense soup.
        {"name": "closest_soup_1m", "kind": "trace", "scene": "soup", "tris": 1_000_000, "rounds": 3,
         "rays": "random", "n": 4_194_304, "mode": "exact", "buffers": "device"},
        # Its any-hit half: shadow rays with a distance limit.
        {"name": "shadow_soup_1m", "kind": "trace", "scene": "soup", "tris": 1_000_000, "rounds": 3,
         "rays": "shadow", "n": 4_194_304, "mode": "exact", "buffers": "device"},
        # A ragged mid-size query job in the compressed 8-wide mode.
        {"name": "closest_fast_ragged", "kind": "trace", "scene": "soup", "tris": 120_011, "rounds": 3,
         "rays": "random", "n": 262_147, "mode": "fast", "buffers": "device"},
        # Coherent primary rays of a full-HD camera over tessellated spheres.
        {"name": "camera_spheres", "kind": "trace", "scene": "spheres", "tris": 1_310_738, "rounds": 3,
         "rays": "camera", "n": 2_073_600, "mode": "exact", "buffers": "device"},
        # A query job from host memory: copies and traversal overlapped.
        {"name": "closest_host", "kind": "trace", "scene": "soup", "tris": 200_003, "rounds": 3, "rays": "random",
         "n": 1_000_003, "mode": "exact", "buffers": "host"},
        # The smallest build, with every node read back.
        {"name": "build_room", "kind": "export", "tris": 36, "rounds": 2},
        # A large scene rebuilt with treelet rounds, then a first batch of shadow rays on the new tree.
        {"name": "frame_soup_1m", "kind": "frame", "tris": 1_000_000, "rounds": 3, "rays": "shadow", "n": 65_536,
         "mode": "exact"},
        # Many small scenes admitted together by a server: one batched build.
        {"name": "batch_48", "kind": "batch", "scenes": 48, "least": 1000, "most": 30_000, "rounds": 3, "n": 2048},
        # The small room rendered whole, plain path integrator.
        {"name": "render_room", "kind": "render", "scene": "room", "size": 0, "width": 256, "height": 256, "spp": 16,
         "depth": 5, "fast": False},
        # A large scene with all four materials, deep paths.
        {"name": "render_spheres", "kind": "render", "scene": "spheres", "size": 5, "width": 1280, "height": 720,
         "spp": 8, "depth": 8, "fast": False},
        # One training batch of the learned proposal (the guided integrator's batch size): loss and gradients.
        {"name": "mlp_gradients", "kind": "mlp", "pass": "gradients", "n": 16_384},
    ]


def _between(rng, lo: float, hi: float) -> int:
    """Log-uniform whole number in [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["trace", "trace", "trace", "frame", "batch", "render", "render", "mlp"])
    if kind == "trace":
        scene = rng.choice(["soup", "soup", "room", "spheres"])
        rays = rng.choice(["random", "shadow"] + (["camera"] if scene == "spheres" else []))
        n = _between(rng, 1000, 4_000_000)
        mode = rng.choice(["exact", "exact", "fast"])
        if scene == "room":  # the exact mode only: nobody needs the 8-wide view of 36 triangles
            tris, mode = 36, "exact"
        elif scene == "spheres":
            tris = 64 * 20 * 4 ** rng.randint(2, 5) + 18
        else:
            tris = _between(rng, 1000, 1_000_000)
        return {"kind": "trace", "scene": scene, "tris": tris, "rounds": rng.choice([0, 3]), "rays": rays, "n": n,
                "mode": mode, "buffers": rng.choice(["device", "device", "host"])}
    if kind == "frame":
        return {"kind": "frame", "tris": _between(rng, 100, 1_000_000), "rounds": rng.choice([0, 1, 3]),
                "rays": rng.choice(["random", "shadow"]), "n": _between(rng, 1000, 300_000),
                "mode": rng.choice(["exact", "exact", "fast"])}
    if kind == "batch":
        least = _between(rng, 100, 3000)
        return {"kind": "batch", "scenes": rng.randint(4, 60), "least": least, "most": least * rng.randint(2, 20),
                "rounds": rng.choice([0, 1, 3]), "n": _between(rng, 256, 4096)}
    if kind == "render":
        scene = rng.choice(["room", "spheres", "soup"])
        size = {"room": 0, "spheres": rng.randint(2, 5), "soup": _between(rng, 1000, 200_000)}[scene]
        return {"kind": "render", "scene": scene, "size": size, "width": rng.randint(64, 640),
                "height": rng.randint(64, 480), "spp": rng.choice([1, 2, 4, 8]), "depth": rng.randint(2, 8),
                "fast": scene != "room" and rng.random() < 0.4}
    if rng.random() < 0.5:
        return {"kind": "mlp", "pass": "forward", "n": _between(rng, 1000, 2_000_000)}
    return {"kind": "mlp", "pass": "gradients", "n": _between(rng, 1000, 65_536)}


# ------------------------------------------------------------------------------ inputs
def _gen(seed: int, salt: int = 0) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + salt)


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _directions(g, n):
    z = 2.0 * _rand(g, n) - 1.0
    phi = 2.0 * math.pi * _rand(g, n)
    r = torch.sqrt(torch.clamp(1.0 - z * z, min=0.0))
    return torch.stack([r * torch.cos(phi), r * torch.sin(phi), z], 1)


def _soup(n: int, g):
    """``scenes.soup`` on the GPU: anchors uniform in the unit cube, vertex offsets of
    log-uniform length in [1e-3, 1e-1]."""
    anchor = _rand(g, n, 1, 3)
    length = torch.exp(math.log(1e-3) + (math.log(1e-1) - math.log(1e-3)) * _rand(g, n, 3, 1))
    pos = (anchor + _directions(g, 3 * n).view(n, 3, 3) * length).to(torch.float32).view(3 * n, 3).contiguous()
    return pos, torch.arange(3 * n, device="cuda", dtype=torch.int32).view(n, 3)


def _sphere_scene(tris: int, seed: int) -> dict:
    level = round(math.log((tris - 18) / (64 * 20), 4))
    return scenes.sphere_scene(64, level, seed=seed % 1000)


def _geometry(case, seed):
    """(positions, indices) on the GPU and the box that ray origins are drawn from."""
    if case.get("scene", "soup") == "soup":
        pos, idx = _soup(case["tris"], _gen(seed))
        return pos, idx, (-0.1, 1.1)
    sc = scenes.mini_room() if case["scene"] == "room" else _sphere_scene(case["tris"], seed)
    lo, hi = sc["positions"].min(0), sc["positions"].max(0)
    return torch.from_numpy(sc["positions"]).cuda(), torch.from_numpy(sc["indices"]).cuda(), (lo, hi)


def _records(o, d):
    n = o.shape[0]
    rays = torch.zeros((n, 8), device="cuda", dtype=torch.float32)
    rays[:, 0:3] = o
    rays[:, 4:7] = d
    rays[:, 7] = math.inf
    return rays


def _rays(kind: str, n: int, box, seed: int):
    """(rays [n, 8], limit [n] or None) on the GPU."""
    g = _gen(seed, 1)
    lo = torch.as_tensor(np.broadcast_to(np.asarray(box[0], np.float64), 3).copy(), device="cuda")
    hi = torch.as_tensor(np.broadcast_to(np.asarray(box[1], np.float64), 3).copy(), device="cuda")
    if kind == "camera":  # a jittered 16:9 pinhole grid from near the front wall, looking inwards
        w = max(1, int(math.sqrt(n * 16 / 9)))
        h = -(-n // w)
        i = torch.arange(n, device="cuda", dtype=torch.float64)
        x = ((i % w) + _rand(g, n)) / w * 2 - 1
        y = 1 - (torch.div(i, w, rounding_mode="floor") + _rand(g, n)) / h * 2
        t = math.tan(math.radians(30.0))
        d = torch.stack([x * t * 16 / 9, y * t, torch.ones_like(x)], 1)
        d = d / torch.linalg.vector_norm(d, dim=1, keepdim=True)
        mid = 0.5 * (lo + hi)
        eye = torch.stack([mid[0], mid[1], lo[2] + 0.025 * (hi[2] - lo[2])])
        return _records(eye.expand(n, 3), d), None
    o = lo + (hi - lo) * _rand(g, n, 3)
    if kind == "random":
        return _records(o, _directions(g, n)), None
    o = o.to(torch.float32).double()
    inner = (0.0, 1.0) if box[0] is not None and np.ndim(box[0]) == 0 else None
    p = _rand(g, n, 3) if inner else lo + (hi - lo) * _rand(g, n, 3)
    v = p - o
    dist = torch.clamp(torch.linalg.vector_norm(v, dim=1), min=1e-6).to(torch.float32)
    return _records(o, v / dist[:, None].double()), dist.contiguous()


def _network(seed: int) -> np.ndarray:
    """Parameters of a network that has left its initial state: Xavier-uniform weights, small
    biases, lobes spread by the last bias."""
    rng = np.random.default_rng(seed)
    parts = []
    for i, o in ((160, 64), (64, 64), (64, 64), (64, 32)):
        a = math.sqrt(6.0 / (i + o))
        parts += [rng.uniform(-a, a, i * o), rng.normal(0.0, 0.5 if o == 32 else 0.05, o)]
    return np.concatenate(parts).astype(np.float32)


def _vertices(n: int, seed: int):
    """Surface points (5 inputs in [0, 1]), directions and radiance weights of n path vertices."""
    g = _gen(seed, 2)
    x = _rand(g, n, 5).to(torch.float32).contiguous()
    d = _directions(g, n).to(torch.float32).contiguous()
    w = (0.1 + 1.9 * _rand(g, n)).to(torch.float32).contiguous()
    return x, d, w


def _load_scene(case, seed):
    """The case's scene written as a .pbrt file and loaded, as a program that renders files does."""
    if case["scene"] == "room":
        sc, ply = scenes.mini_room(), False
        # the room's light differs from seed to seed, its geometry does not
        rng = np.random.default_rng(seed)
        sc["light_radiance"] = tuple(float(v) for v in rng.uniform(4.0, 20.0, 3))
    elif case["scene"] == "spheres":
        sc, ply = scenes.sphere_scene(64, case["size"], seed=seed % 1000), True
    else:
        sc, ply = scenes.soup_scene(case["size"], seed=seed % 1000), True
    with tempfile.TemporaryDirectory() as tmp:
        path = os.path.join(tmp, "scene.pbrt")
        scenes.write_pbrt(path, sc, width=case["width"], height=case["height"], spp=case["spp"],
                          max_depth=case["depth"], ply=ply)
        return _ctx().load_pbrt(path, bvh_rounds=0 if case["scene"] == "room" else 3)


def prepare(case: dict, seed: int):
    kind = case["kind"]
    if kind == "trace":
        pos, idx, box = _geometry(case, seed)
        rays, limit = _rays(case["rays"], case["n"], box, seed)
        bvh = _ctx().build(pos, idx, rounds=case["rounds"])
        if case["buffers"] == "host":  # pinned buffers, kept by the program
            rays = rays.cpu().pin_memory()
            limit = None if limit is None else limit.cpu().pin_memory()
            n = case["n"]
            if limit is None:
                out = (torch.empty(n, dtype=torch.int32).pin_memory(), torch.empty(n).pin_memory(),
                       torch.empty((n, 2)).pin_memory())
            else:
                out = torch.empty(n, dtype=torch.uint8).pin_memory()
        else:
            out = None
        return {"case": case, "bvh": bvh, "rays": rays, "limit": limit, "out": out}
    if kind == "export":
        sc = scenes.mini_room()
        # the whole room scaled by the seed: another size of the same layout
        scale = 1.0 + (seed % 997) / 997.0
        pos = torch.from_numpy(sc["positions"] * np.float32(scale)).cuda()
        return {"case": case, "pos": pos, "idx": torch.from_numpy(sc["indices"]).cuda()}
    if kind == "frame":
        pos, idx, box = _geometry(case, seed)
        rays, limit = _rays(case["rays"], case["n"], box, seed)
        return {"case": case, "pos": pos, "idx": idx, "rays": rays, "limit": limit}
    if kind == "batch":
        rng = np.random.default_rng(seed)
        g = _gen(seed)
        sizes = np.exp(rng.uniform(math.log(case["least"]), math.log(case["most"]), case["scenes"])).astype(int)
        rays, _ = _rays("random", case["n"], (-0.1, 1.1), seed)
        return {"case": case, "scenes": [_soup(int(n), g) for n in sizes], "rays": rays}
    if kind == "render":
        return {"case": case, "scene": _load_scene(case, seed)}
    net = cav.Mlp(_ctx())
    net.set_params(_network(seed))
    x, d, w = _vertices(case["n"], seed)
    return {"case": case, "net": net, "x": x, "d": d, "w": w}


# --------------------------------------------------------------------------------- run
def _query(bvh, rays, limit, mode):
    if limit is not None:
        return bvh.trace_any(rays, limit, flags=_MODES[mode])
    return bvh.trace_closest(rays, flags=_MODES[mode])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "trace":
        bvh, rays, limit = state["bvh"], state["rays"], state["limit"]
        if case["buffers"] == "device":
            return _query(bvh, rays, limit, case["mode"])
        if limit is not None:
            return bvh.trace_any_host(rays, limit, flags=_MODES[case["mode"]], out=state["out"])
        return bvh.trace_closest_host(rays, flags=_MODES[case["mode"]], out=state["out"])
    if kind == "export":
        bvh = _ctx().build(state["pos"], state["idx"], rounds=case["rounds"])
        nodes = bvh.export_nodes()
        codes, ordered, prims = bvh.export_stages()
        bvh.free()
        return {"bmin": nodes["bmin"], "bmax": nodes["bmax"], "left": nodes["left"], "right": nodes["right"],
                "leaf": nodes["is_leaf"], "prim": nodes["prim_begin"], "codes": codes.view(np.int64),
                "ordered": ordered.view(np.int64), "prims": prims}
    if kind == "frame":
        bvh = _ctx().build(state["pos"], state["idx"], rounds=case["rounds"])
        out = _query(bvh, state["rays"], state["limit"], case["mode"])
        bvh.free()
        return out
    if kind == "batch":
        trees = _ctx().build_batch(state["scenes"], rounds=case["rounds"])
        hits = [t.trace_closest(state["rays"]) for t in trees]
        for t in trees:
            t.free()
        return [torch.stack([h[k] for h in hits]) for k in range(3)]
    if kind == "render":
        film, weight, _ = state["scene"].render(fast_trace=case["fast"])
        return film, weight
    if case["pass"] == "forward":
        return state["net"].forward(state["x"])
    return state["net"].gradients(state["x"], state["d"], state["w"])


# -------------------------------------------------------------------------------- work
def work(case: dict) -> dict:
    kind = case["kind"]
    tri = 48.0  # three vertices and three indices, read once
    if kind == "trace":
        n = case["n"]
        # the ray, its limit and its result; the triangles that so many rays can need
        io = 32.0 + (4.0 + 1.0 if case["rays"] == "shadow" else 16.0)
        return {"bytes": n * io + tri * min(n, case["tris"]), "flops": 100.0 * n}
    if kind == "export":
        return {"bytes": case["tris"] * (tri + 2 * 44.0 + 20.0), "flops": 100.0 * case["tris"]}
    if kind == "frame":
        io = 32.0 + (4.0 + 1.0 if case["rays"] == "shadow" else 16.0)
        return {"bytes": case["tris"] * tri + case["n"] * io, "flops": 100.0 * case["tris"]}
    if kind == "batch":
        mean = (case["most"] - case["least"]) / math.log(max(case["most"] / case["least"], 1.0001))
        return {"bytes": case["scenes"] * (mean * tri + case["n"] * 16.0) + 32.0 * case["n"],
                "flops": 100.0 * case["scenes"] * mean}
    if kind == "render":
        pixels = case["width"] * case["height"]
        tris = {"room": 36, "spheres": 64 * 20 * 4 ** case["size"] + 18, "soup": case["size"]}[case["scene"]]
        # the film and the scene; about 500 operations to shade a path's vertex
        return {"bytes": 16.0 * pixels + tri * tris, "flops": 500.0 * pixels * case["spp"] * case["depth"]}
    n = case["n"]
    forward = 2.0 * (160 * 64 + 64 * 64 + 64 * 64 + 64 * 32)
    params = 4.0 * (160 * 64 + 64 + 2 * (64 * 64 + 64) + 64 * 32 + 32)
    if case["pass"] == "forward":
        return {"bytes": n * (20.0 + 128.0) + params, "flops": n * forward}
    # forward, weight gradients, and input gradients of all layers but the first
    return {"bytes": n * 36.0 + 2 * params, "flops": n * (2 * forward + 2.0 * (64 * 64 + 64 * 64 + 64 * 32))}


def tolerance(case: dict):
    kind = case["kind"]
    if kind in ("export", "batch") or case.get("mode") == "exact":
        return "exact"  # the exact mode's hits are those of the reference's traversal, bit for bit
    if kind in ("trace", "frame"):
        # fast mode: the same distances; at a tie (a ray through a shared edge, about one in a
        # million) another triangle, and with it other barycentrics: one such ray in 10^5 is
        # 3e-3 of the norm
        return {"rel": 3e-3, "max": 1.0 - 1e-6, "differ": 1e-4}
    if kind == "render":
        return {"rel": 1e-3, "max": 0.5}  # float film sums in another order
    if case["pass"] == "forward":
        return {"rel": 2e-3, "max": 2e-2}  # BF16 activations
    return {"rel": 1e-2, "max": 0.3}  # BF16 activations and back-propagated gradients


# ------------------------------------------------------------------------------- exact
def _nearest(pos, idx, rays):
    """Closest-hit distances in 64 bits by testing every triangle (inf on a miss)."""
    p = pos.double()
    v0, v1, v2 = (p[idx[:, k].long()] for k in range(3))
    e1, e2 = v1 - v0, v2 - v0
    out = torch.full((rays.shape[0],), math.inf, device="cuda", dtype=torch.float64)
    step = max(1, 8_000_000 // idx.shape[0])
    for at in range(0, rays.shape[0], step):
        r = rays[at:at + step].double()
        o, d = r[:, None, 0:3], r[:, None, 4:7]
        tv = o - v0
        pv = torch.cross(d.expand_as(tv), e2.expand_as(tv), dim=2)
        det = (e1 * pv).sum(2)
        u = (tv * pv).sum(2) / det
        qv = torch.cross(tv, e1.expand_as(tv), dim=2)
        v = (d * qv).sum(2) / det
        t = (e2 * qv).sum(2) / det
        hit = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0)
        out[at:at + step] = torch.where(hit, t, math.inf).min(1).values
    return out


def _layers(params):
    p = torch.from_numpy(params).double().cuda()
    at, out = 0, []
    for i, o in ((160, 64), (64, 64), (64, 64), (64, 32)):
        out += [p[at:at + i * o].view(o, i), p[at + i * o:at + i * o + o]]
        at += i * o + o
    return out


def _forward64(layers, x):
    centres = (torch.arange(32, device="cuda", dtype=torch.float64) + 0.5) / 32
    h = torch.exp(-0.5 * ((x.double()[:, :, None] - centres) * 32) ** 2).reshape(len(x), 160)
    for k in range(4):
        h = h @ layers[2 * k].T + layers[2 * k + 1]
        if k < 3:
            h = torch.relu(h)
    return h


def _loss64(out, d, w):
    """mean(-w log q(d)) of the 8-lobe von Mises-Fisher mixture."""
    o = out.view(-1, 8, 4)
    pi = torch.softmax(o[..., 0], 1)
    th, ph = math.pi * torch.sigmoid(o[..., 1]), 2 * math.pi * torch.sigmoid(o[..., 2])
    mu = torch.stack([torch.sin(th) * torch.cos(ph), torch.sin(th) * torch.sin(ph), torch.cos(th)], -1)
    kappa = torch.clamp(torch.nn.functional.softplus(o[..., 3]) + 0.01, max=500.0)
    norm = kappa / (2 * math.pi * (1 - torch.exp(-2 * kappa)))
    c = (mu * d.double()[:, None, :]).sum(-1)
    q = (pi * norm * torch.exp(kappa * (c - 1))).sum(1)
    return -(w.double() * torch.log(q)).mean()


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("trace", "frame") and case["rays"] != "shadow" and case["n"] * case["tris"] <= 2e9:
        pos, idx, box = _geometry(case, seed)
        rays, _ = _rays(case["rays"], case["n"], box, seed)
        return None, _nearest(pos, idx, rays), None
    if kind == "mlp":
        layers = [t.requires_grad_(case["pass"] == "gradients") for t in _layers(_network(seed))]
        x, d, w = _vertices(case["n"], seed)
        if case["pass"] == "forward":
            return _forward64(layers, x) if case["n"] <= 500_000 else None
        loss = _loss64(_forward64(layers, x), d, w)
        grads = torch.autograd.grad(loss, layers)
        return torch.cat([g.reshape(-1) for g in grads]).cpu().numpy(), float(loss)
    return None
