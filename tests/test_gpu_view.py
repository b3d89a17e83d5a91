"""GPU tests of how a tree's 8-wide view comes about in the exact mode: enqueued by the query that
has asked about enough rays, waited for by nobody, done without where there is no memory for it
or the stream is being captured.  Answers are the binary traversal's throughout."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BINARY = (1 << 22) - 1  # one below the default limit: the same answers from the binary traversal


def _tree(ctx, n, seed=3, rays=20_000):
    import torch

    from cavalry_b200 import scenes

    pos, idx = scenes.soup(n, seed=seed)
    bvh = ctx.build(torch.from_numpy(pos).cuda(), torch.from_numpy(idx).cuda(), rounds=1)
    shadow, limit = scenes.shadow_rays(rays, seed=seed + 1)
    return (bvh, torch.from_numpy(scenes.closest_rays(rays, seed=seed)).cuda(), torch.from_numpy(shadow).cuda(),
            torch.from_numpy(limit).cuda())


def _same(got, want):
    import torch

    return all(torch.equal(g.view(torch.uint8), w.view(torch.uint8)) for g, w in zip(got, want))


def _binary(ctx, bvh, rays, shadow, limit):
    import torch

    ctx.set_limits(max_trace_steps=BINARY)
    want = [*bvh.trace_closest(rays), bvh.trace_any(shadow, limit)]
    ctx.set_limits()
    torch.cuda.synchronize()
    return want


def test_a_query_that_begins_the_view_waits_for_nothing():
    """Behind half a second of other work on its stream the first queries return at once, and one
    on another stream is answered meanwhile, before the view that it cannot use yet."""
    import torch

    import cavalry_b200 as cav

    ctx = cav.Context(0)
    try:
        warm, rays, shadow, limit = _tree(ctx, 30_000, seed=9)  # modules loaded, memory pool grown
        for _ in range(2):
            warm.trace_closest(rays), warm.trace_any(shadow, limit)
        warm.trace_closest(rays, flags=cav.TRACE_FAST)
        torch.cuda.synchronize()
        bvh, rays, shadow, limit = _tree(ctx, 30_000)
        want = _binary(ctx, bvh, rays, shadow, limit)
        assert not bvh.has_fast_layout()
        a, b = torch.cuda.Stream(), torch.cuda.Stream()
        # outputs exist beforehand: the caching allocator is not what is tested
        outs = [(torch.empty(len(rays), dtype=torch.int32, device="cuda"), torch.empty(len(rays), device="cuda"),
                 torch.empty((len(rays), 2), device="cuda"), torch.empty(len(rays), dtype=torch.uint8, device="cuda"))
                for _ in range(2)]
        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            torch.cuda._sleep(1_000_000_000)
        for s, o in ((a, outs[0]), (b, outs[1])):
            bvh.trace_closest(rays, stream=s, out=o[:3])
            bvh.trace_any(shadow, limit, stream=s, out=o[3])
            if s is a:
                assert bvh.has_fast_layout()  # begun
        b.synchronize()
        assert not a.query()
        assert _same(outs[1], want)
        a.synchronize()
        assert _same(outs[0], want)
        assert _same([*bvh.trace_closest(rays), bvh.trace_any(shadow, limit)], want)
        ctx.sync_check()
        bvh.free(), warm.free()
    finally:
        ctx.close()


def test_no_memory_for_the_view():
    """The query succeeds without it, and a later one has it."""
    import cavalry_b200 as cav

    ctx = cav.Context(0)
    try:
        bvh, rays, shadow, limit = _tree(ctx, 30_000)
        want = _binary(ctx, bvh, rays, shadow, limit)
        ctx.inject(cav.INJECT_ALLOC_FAIL, 1)
        assert _same(bvh.trace_closest(rays), want)
        assert not bvh.has_fast_layout()
        assert _same([bvh.trace_any(shadow, limit)], want[3:])  # asked about more than twice 512 rays
        assert bvh.has_fast_layout()
        assert _same([*bvh.trace_closest(rays), bvh.trace_any(shadow, limit)], want)
        ctx.sync_check()
        bvh.free()
    finally:
        ctx.inject(cav.INJECT_NONE)
        ctx.close()


@pytest.mark.parametrize("view", [False, True])
def test_a_stream_in_capture(view):
    """A captured query takes the view that is complete, or the binary traversal."""
    import torch

    import cavalry_b200 as cav

    ctx = cav.Context(0)
    try:
        bvh, rays, shadow, limit = _tree(ctx, 30_000)
        want = _binary(ctx, bvh, rays, shadow, limit)
        if view:
            bvh.trace_any(shadow, limit)
            torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            got = [*bvh.trace_closest(rays), bvh.trace_any(shadow, limit)]
        assert bool(bvh.has_fast_layout()) == view
        for o in got:
            o.fill_(1)
        g.replay()
        torch.cuda.synchronize()
        assert _same(got, want)
        ctx.sync_check()
        del g
        bvh.free()
    finally:
        ctx.close()


@pytest.mark.parametrize("batch", [False, True])
def test_threads_that_reach_first_views_together(batch):
    """Four threads, each with a context and a stream of its own, query the same trees, the fast
    mode (which waits for the view) among them; trees are freed while others are still queried."""
    import torch

    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    main = cav.Context(0)
    ctxs = [cav.Context(0) for _ in range(4)]
    try:
        geo = [scenes.soup(n, seed=n) for n in (5000, 9001, 200, 30_000)]
        geo = [(torch.from_numpy(p).cuda(), torch.from_numpy(i).cuda()) for p, i in geo]
        trees = main.build_batch(geo, rounds=1) if batch else [main.build(p, i, rounds=1) for p, i in geo]
        rays = torch.from_numpy(scenes.closest_rays(20_000, seed=5)).cuda()
        main.set_limits(max_trace_steps=BINARY)
        want = [t.trace_closest(rays) for t in trees]
        main.set_limits()
        torch.cuda.synchronize()
        bad, gate = [], threading.Barrier(4)

        def work(k):
            try:
                s = torch.cuda.Stream()
                gate.wait()
                with torch.cuda.stream(s):
                    for r in range(6):
                        for j, t in enumerate(trees):
                            b = cav.Bvh(ctxs[k], t.handle, t.n, owned=False)  # through this thread's context
                            if k == 3 and r == 2:
                                dist = b.trace_closest(rays, flags=cav.TRACE_FAST)[1]
                                s.synchronize()
                                if not torch.equal(dist, want[j][1]):
                                    bad.append((k, j, "fast"))
                            got = b.trace_closest(rays)
                            s.synchronize()
                            if not _same(got, want[j]):
                                bad.append((k, r, j))
                ctxs[k].sync_check()
            except Exception as e:  # noqa: BLE001
                bad.append((k, repr(e)))

        ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert bad == []
        for t in trees[:2]:
            t.free()
        got = [t.trace_closest(rays) for t in trees[2:]]
        assert all(_same(g, w) for g, w in zip(got, want[2:]))
        for t in trees[2:]:
            t.free()
        main.sync_check()
    finally:
        for c in ctxs:
            c.close()
        main.close()


def test_a_view_with_a_node_for_each_binary_node():
    """Flat boxes of infinite extent have no area to open by, so every wide node holds two children:
    more nodes than finite geometry can have.  The fast mode still gets its view, alone and in a
    batch, and the exact mode's answers stay the binary traversal's."""
    import torch

    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    ctx = cav.Context(0)
    try:
        n = 600
        pos = np.zeros((3 * n, 3), np.float32)
        pos[0::3, 0], pos[1::3, 0] = -np.inf, np.inf
        pos[2::3, 1] = np.linspace(0.0, 1.0, n)
        pos[:, 1] = np.repeat(pos[2::3, 1], 3)  # each in a plane of its own, flat in y
        idx = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
        geo = (torch.from_numpy(pos).cuda(), torch.from_numpy(idx).cuda())
        other = tuple(torch.from_numpy(a).cuda() for a in scenes.soup(5000, seed=1))
        rays = torch.from_numpy(scenes.closest_rays(20_000, seed=2)).cuda()
        trees = [ctx.build(*geo, rounds=0), *ctx.build_batch([geo, other], rounds=0)]
        for t in trees:
            ctx.set_limits(max_trace_steps=BINARY)
            want = t.trace_closest(rays)
            ctx.set_limits()
            for _ in range(2):
                assert _same(t.trace_closest(rays), want)
                assert torch.equal(t.trace_closest(rays, flags=cav.TRACE_FAST)[1], want[1])
            assert t.has_fast_layout()
            assert _same(t.trace_closest(rays), want)
        ctx.sync_check()
        for t in trees:
            t.free()
    finally:
        ctx.close()


@pytest.mark.parametrize("scene,n", [("soup", 2**21 - 1), ("soup", 2**21), ("soup", 2**21 + 3), ("spheres", 2**19 - 1),
                                     ("spheres", 2**19 + 3)])
def test_host_calls_at_their_first_view(scene, n):
    """Closest hits from pageable buffers below, at and above the sizes where they are cut into two
    chunks (2^20 rays each in the binary traversal, 2^18 through the view), on a tree whose first call
    begins the view and on the same tree with the view: the device call's results."""
    import torch

    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    ctx = cav.Context(0)
    try:
        if scene == "soup":
            pos, idx = scenes.soup(40_000, seed=6)
        else:
            s = scenes.sphere_scene(8, 2, seed=6)
            pos, idx = s["positions"], s["indices"]
        geo = (torch.from_numpy(pos).cuda(), torch.from_numpy(idx).cuda())
        rays = scenes.closest_rays(n, seed=7)
        shadow, limit = scenes.shadow_rays(n, seed=8)
        want = None
        for first in (True, False):
            bvh = ctx.build(*geo, rounds=2)
            if want is None:
                ctx.set_limits(max_trace_steps=BINARY)
                want = [a.cpu().numpy() for a in bvh.trace_closest(torch.from_numpy(rays).cuda())]
                occ = bvh.trace_any(torch.from_numpy(shadow).cuda(), torch.from_numpy(limit).cuda()).cpu().numpy()
                ctx.set_limits()
            if not first:
                bvh.trace_any(torch.from_numpy(shadow).cuda())
                torch.cuda.synchronize()
                assert bvh.has_fast_layout()
                bvh.trace_any(torch.from_numpy(shadow).cuda())
            got = bvh.trace_closest_host(rays)
            assert all(np.array_equal(g.view(np.uint8), w.view(np.uint8)) for g, w in zip(got, want))
            assert np.array_equal(bvh.trace_any_host(shadow, limit), occ)
            ctx.sync_check()
            bvh.free()
    finally:
        ctx.close()


@pytest.mark.parametrize("dense", [False, True])
def test_graph_renders_with_and_without_a_view(dense, tmp_path):
    """An exact graph render captures the view's launches where the view is complete, with the binary
    ones beside them where only the device knows which serve the rays (densely overlapping boxes), and
    the binary ones where there is no view: the stream-ordered render's film and ray counts."""
    import torch

    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    ctx = cav.Context(0)
    try:
        s = scenes.soup_scene(40_000, seed=4) if dense else scenes.sphere_scene(8, 2, seed=5)
        path = str(tmp_path / "scene.pbrt")
        scenes.write_pbrt(path, s, width=96, height=64, spp=4, max_depth=5, ply=True)
        sc = ctx.load_pbrt(path, bvh_rounds=2)
        bvh = sc.bvh()
        nodes = bvh.export_nodes()
        e = (nodes["bmax"] - nodes["bmin"]).astype(np.float64)
        area = e[:, 0] * e[:, 1] + e[:, 1] * e[:, 2] + e[:, 2] * e[:, 0]
        lines = area[nodes["is_leaf"].astype(bool)].sum() / area[0]
        assert lines > 13 if dense else lines < 11  # the rule's line is at 12
        films, counts = [], []
        rays = torch.from_numpy(scenes.closest_rays(20_000, seed=1)).cuda()
        for view in (False, True):
            if view:
                bvh.trace_any(rays)
                torch.cuda.synchronize()
                assert bvh.has_fast_layout()
            f, w, _ = sc.render(graph=True)
            films.append((f, w))
            counts.append((sc.stats().closest_rays, sc.stats().shadow_rays))
            assert bool(bvh.has_fast_layout()) == view
        f, w, _ = sc.render()
        films.append((f, w))
        counts.append((sc.stats().closest_rays, sc.stats().shadow_rays))
        assert counts[0] == counts[1] == counts[2] and counts[0][0] > 20_000
        for f, w in films[1:]:
            assert np.array_equal(w, films[0][1])
            assert np.allclose(f, films[0][0], rtol=2e-5, atol=1e-6)  # float film sums in another order
        ctx.sync_check()
        del sc, bvh
    finally:
        ctx.close()
