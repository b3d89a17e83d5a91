"""GPU tests of the exact mode through the compressed 8-wide view (the screening pass): hits,
distances and barycentrics bit for bit those of the binary traversal on the same tree, which a
lowered step limit still selects."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BINARY = (1 << 22) - 1  # one below the default limit: the same answers from the binary traversal


def rays_for(kind, pos, idx, n, rng):
    from cavalry_b200 import scenes

    lo, hi = pos.min(0), pos.max(0)
    o = rng.uniform(lo - 0.1 * (hi - lo), hi + 0.1 * (hi - lo), (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    if kind == "axis":  # one or two zero components, either sign
        z = rng.integers(0, 3, n)
        d[np.arange(n), z] = np.where(rng.random(n) < 0.5, 0.0, -0.0)
        two = rng.random(n) < 0.3
        d[two, (z[two] + 1) % 3] = 0.0
    if kind == "edges":  # through shared edges and vertices: ties of two and more
        t = idx[rng.integers(0, len(idx), n)]
        w = rng.random((n, 1)).astype(np.float32)
        w[: n // 3] = 1.0
        d = (pos[t[:, 0]] * w + pos[t[:, 1]] * (1 - w) - o).astype(np.float32)
    r = scenes.make_rays(o, d)
    if kind == "odd":  # values the screening refuses or must not trip over
        bad = np.array([np.nan, np.inf, -np.inf, 1e-38, 1e-45, 3e38, 0.0], np.float32)
        k = rng.integers(0, n, n // 4)
        r[k, rng.integers(0, 8, len(k))] = bad[rng.integers(0, len(bad), len(k))]
        r[::3, 7] = rng.random(len(r[::3]))
    return r


def geometry(name, n, rng):
    from cavalry_b200 import scenes

    if name == "spheres":
        s = scenes.sphere_scene(8, n, seed=5)
        return s["positions"], s["indices"]
    pos, idx = scenes.soup(n, seed=int(rng.integers(1 << 30)))
    if name == "duplicates":  # every triangle twice, with opposite winding: every hit is a tie
        idx = np.ascontiguousarray(np.concatenate([idx, idx[:, ::-1]]))
    if name == "far":  # boxes a few ulps of the coordinates wide
        pos = (pos + np.float32(3000.0)).astype(np.float32)
    if name == "nan":
        pos = pos.copy()
        pos[::97, 1] = np.nan
    return pos, idx


@pytest.mark.parametrize("name,size,n", [
    ("soup", 129, 20_001), ("soup", 4096, 512), ("soup", 4097, 70_001), ("soup", 60_000, 262_147), ("spheres", 2, 33_333),
    ("spheres", 4, 200_000), ("duplicates", 3000, 50_000), ("far", 5000, 50_000), ("nan", 5000, 30_000)])
def test_screened_hits_are_the_binary_traversals(name, size, n):
    """Below and above a warp's share of the rays, the thresholds of the view, and every kind of
    ray that is proven, searched again or handed to the binary steps."""
    import torch

    import cavalry_b200 as cav

    rng = np.random.default_rng(size + n)
    pos, idx = geometry(name, size, rng)
    mesh = (np.arange(len(idx)) % 5).astype(np.int32)
    gpu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    ctx = cav.Context(0)
    try:
        bvh = ctx.build(gpu(pos), gpu(idx), gpu(mesh), rounds=2)
        for kind in ("random", "axis", "edges", "odd"):
            if name == "nan" and kind == "edges":
                continue
            r = rays_for(kind, np.nan_to_num(pos), idx, n, rng)
            lim = (rng.random(n) * 0.7).astype(np.float32)
            ex = rng.integers(-1, 5, (n, 2)).astype(np.int32)
            r, lim, ex = gpu(r), gpu(lim), gpu(ex)
            got = [*bvh.trace_closest(r), bvh.trace_any(r, lim), bvh.trace_any(r, lim, ex), bvh.trace_any(r)]
            assert bvh.has_fast_layout()
            ctx.set_limits(max_trace_steps=BINARY)
            want = [*bvh.trace_closest(r), bvh.trace_any(r, lim), bvh.trace_any(r, lim, ex), bvh.trace_any(r)]
            ctx.set_limits()
            for k, (g, w) in enumerate(zip(got, want)):
                assert torch.equal(g.view(torch.uint8), w.view(torch.uint8)), (kind, k)
        ctx.sync_check()
        bvh.free()
    finally:
        ctx.close()


@pytest.mark.parametrize("size", [2, 3, 8, 9, 36, 65, 128, 1000, 1025])
@pytest.mark.parametrize("n", [1, 4, 31, 5000])
def test_small_views_and_batches(size, n):
    """Views of one node, one block and several; batches below, at and above a warp's smallest
    share of rays: the fast mode's distances and any-hit answers are the exact mode's."""
    import torch

    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    ctx = cav.Context(0)
    try:
        pos, idx = scenes.soup(size, seed=size)
        bvh = ctx.build(torch.from_numpy(pos).cuda(), torch.from_numpy(idx).cuda(), rounds=1)
        rng = np.random.default_rng(n)
        t = idx[rng.integers(0, size, n)]  # aimed at triangles, so that most rays hit
        o = rng.uniform(-0.1, 1.1, (n, 3)).astype(np.float32)
        r = torch.from_numpy(scenes.make_rays(o, (pos[t].mean(1) - o).astype(np.float32))).cuda()
        pe, te, _ = bvh.trace_closest(r)
        pf, tf, _ = bvh.trace_closest(r, flags=cav.TRACE_FAST)
        assert torch.equal(pe, pf) and torch.equal(te, tf) and int((pe >= 0).sum()) >= n * 0.9
        lim = torch.full((n,), 0.9, device="cuda")
        assert torch.equal(bvh.trace_any(r, lim), bvh.trace_any(r, lim, flags=cav.TRACE_FAST))
        ctx.sync_check()
        bvh.free()
    finally:
        ctx.close()


def plane_rays(name, n, rng):
    """Rays whose lines lie in triangles' planes, where the triangle test's determinant and distance
    are rounding noise: lines of sight between points of one tilted wall, and rays laid in the
    planes of a soup's or of spheres' triangles, from anywhere in them."""
    from cavalry_b200 import scenes

    if name.startswith("wall"):
        g, off = int(name[4:]), 5.0 if n & 1 else 0.0
        i = np.arange(g + 1) / g
        x, y = (a.ravel()[:, None] for a in np.meshgrid(i, i))
        up = np.array([0.3, 0.5, 0.8]) / np.linalg.norm([0.3, 0.5, 0.8])
        ux = np.cross(up, [0.0, 0.0, 1.0])
        ux /= np.linalg.norm(ux)
        uy = np.cross(up, ux)
        pos = (x * ux + y * uy + off).astype(np.float32)
        q = (np.arange(g)[:, None] * (g + 1) + np.arange(g)).ravel()
        idx = np.concatenate([np.stack([q, q + 1, q + g + 1], 1), np.stack([q + 1, q + g + 2, q + g + 1], 1)])
        a, b = rng.random((2, n, 2))
        o = (a[:, :1] * ux + a[:, 1:] * uy + off).astype(np.float32)
        p = (b[:, :1] * ux + b[:, 1:] * uy + off).astype(np.float32)
    else:
        pos, idx = geometry(name, 5000 if name == "soup" else 3, rng)
        t = idx[rng.integers(0, len(idx), n)]
        v0, v1, v2 = (pos[t[:, k]].astype(np.float64) for k in range(3))
        a, b = rng.uniform(-6, 7, (n, 2)), rng.uniform(-1, 2, (n, 2))
        o = (v0 + a[:, :1] * (v1 - v0) + a[:, 1:] * (v2 - v0)).astype(np.float32)
        p = v0 + b[:, :1] * (v1 - v0) + b[:, 1:] * (v2 - v0)
    d = p - o
    length = np.maximum(np.linalg.norm(d, axis=1), 1e-20)
    rays = scenes.make_rays(o, (d / length[:, None]).astype(np.float32))
    return pos, np.ascontiguousarray(idx, np.int32), rays, (length * 0.999).astype(np.float32)


@pytest.mark.parametrize("name,n", [("wall9", 100_000), ("wall32", 100_001), ("wall128", 200_001), ("soup", 1_000_000),
                                    ("spheres", 1_000_000)])
def test_any_hits_of_rays_in_triangle_planes(name, n):
    """Bit for bit the binary traversal's, with a limit and without."""
    import torch

    import cavalry_b200 as cav

    pos, idx, rays, limit = plane_rays(name, n, np.random.default_rng(n))
    gpu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    ctx = cav.Context(0)
    try:
        bvh = ctx.build(gpu(pos), gpu(idx), rounds=2)
        r, lim = gpu(rays), gpu(limit)
        limits = [lim, 0.3 * lim, None]
        got = [bvh.trace_any(r, x) for x in limits]
        assert bvh.has_fast_layout()
        ctx.set_limits(max_trace_steps=BINARY)
        want = [bvh.trace_any(r, x) for x in limits]
        assert 0.02 * n < int(want[0].sum()) < 0.999 * n
        for g, w in zip(got, want):
            assert int((g != w).sum()) == 0
        ctx.sync_check()
        bvh.free()
    finally:
        ctx.close()


@pytest.mark.parametrize("name,n", [("wall32", 100_001), ("wall128", 150_000), ("soup", 100_000), ("soup", 1_000_000),
                                    ("spheres", 1_000_000)])
def test_closest_hits_of_rays_in_triangle_planes(name, n):
    """Bit for bit the binary traversal's, through the view (few rays, or boxes that overlap little)
    and past it, with a distance bound on part of the rays."""
    import torch

    import cavalry_b200 as cav

    pos, idx, rays, limit = plane_rays(name, n, np.random.default_rng(n + 1))
    rays[::3, 7] = 0.8 * limit[::3]
    gpu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    ctx = cav.Context(0)
    try:
        bvh = ctx.build(gpu(pos), gpu(idx), rounds=2)
        r = gpu(rays)
        bvh.trace_closest(r)
        got = bvh.trace_closest(r)
        assert bvh.has_fast_layout()
        ctx.set_limits(max_trace_steps=BINARY)
        want = bvh.trace_closest(r)
        assert int((want[0] >= 0).sum()) > 0.02 * n
        for g, w in zip(got, want):
            assert torch.equal(g.view(torch.uint8), w.view(torch.uint8))
        ctx.sync_check()
        bvh.free()
    finally:
        ctx.close()
