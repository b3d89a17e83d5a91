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
