"""GPU test of the batched build (cav_bvh_build_batch): every tree equals the tree built
for its scene alone, bit for bit, and traces the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rounds", [0, 2])
def test_batch_build_equals_single_builds(rounds):
    import torch

    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    ctx = cav.Context(0)
    sizes = [2, 3, 1000, 600000, 4097, 33000, 250000, 17]  # 600k: a tree that runs its rounds alone
    data = [scenes.soup(n, seed=40 + k) for k, n in enumerate(sizes)]
    room = scenes.mini_room()
    data.append((room["positions"], room["indices"]))
    dev = [(torch.from_numpy(p).cuda(), torch.from_numpy(i).cuda()) for p, i in data]
    batch = ctx.build_batch(dev, rounds=rounds)
    rays = torch.from_numpy(scenes.closest_rays(20000, seed=5)).cuda()
    for k, (p, i) in enumerate(dev):
        single = ctx.build(p, i, rounds=rounds)
        a, b = batch[k].export_nodes(), single.export_nodes()
        assert a.tobytes() == b.tobytes(), k
        sa, sb = batch[k].export_stages(), single.export_stages()
        for x, y in zip(sa, sb):
            assert np.array_equal(x, y), k
        pa, ta, _ = batch[k].trace_closest(rays)
        pb, tb, _ = single.trace_closest(rays)
        assert np.array_equal(pa.cpu().numpy(), pb.cpu().numpy())
        single.free()
    ctx.sync_check()


def test_many_small_scenes_with_treelet_rounds():
    """96 scenes of 2-6000 triangles with 3 treelet rounds: the rounds run for all trees in
    one leaf-list and one treelet launch per round, and every tree is still the one its
    scene builds alone."""
    import torch

    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    ctx = cav.Context(0)
    rng = np.random.default_rng(12)
    sizes = [2, 3, 4, 5] + [int(x) for x in np.exp(rng.uniform(np.log(6), np.log(6000), 92))]
    dev = []
    for k, n in enumerate(sizes):
        p, i = scenes.soup(n, seed=300 + k)
        dev.append((torch.from_numpy(p).cuda(), torch.from_numpy(i).cuda()))
    batch = ctx.build_batch(dev, rounds=3)
    for k, (p, i) in enumerate(dev):
        single = ctx.build(p, i, rounds=3)
        assert batch[k].export_nodes().tobytes() == single.export_nodes().tobytes(), (k, sizes[k])
        single.free()
    ctx.sync_check()


def test_trees_freed_while_they_are_traced():
    """Trees freed right after their queries were launched, and others of other sizes built at
    once, on the default and on a side stream: the memory is given back only once the queries
    are through, so their hits are those of trees that were kept."""
    import torch

    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    ctx = cav.Context(0)
    rays = torch.from_numpy(scenes.closest_rays(200_000, seed=6)).cuda()
    groups = []
    for g, sizes in enumerate([[30000, 2000, 500], [9000, 15000, 700, 41], [60000, 130]]):
        data = [scenes.soup(n, seed=70 + 10 * g + k) for k, n in enumerate(sizes)]
        groups.append([(torch.from_numpy(p).cuda(), torch.from_numpy(i).cuda()) for p, i in data])
    want = []
    for dev in groups:
        trees = ctx.build_batch(dev, rounds=1)
        want.append([t.trace_closest(rays) for t in trees])
        ctx.sync_check()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for stream in (torch.cuda.current_stream(), side):
        with torch.cuda.stream(stream):
            got = []
            for _ in range(3):
                for dev in groups:
                    trees = ctx.build_batch(dev, rounds=1)
                    got.append([t.trace_closest(rays) for t in trees])
                    for t in trees:
                        t.free()
                    p, i = dev[0]
                    one = ctx.build(p, i, rounds=1)
                    got[-1].append(one.trace_closest(rays))
                    one.free()
        torch.cuda.synchronize()
        for at, hits in enumerate(got):
            ref = want[at % len(groups)]
            for a, b in zip(hits, ref + ref[:1]):
                assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    ctx.sync_check()


@pytest.mark.parametrize("sizes", [[65536, 65537, 2, 300], [129], [65537, 200, 70000], [2, 3, 128, 129, 2000]])
def test_views_of_a_batch_equal_single_views(sizes):
    """The 8-wide views of a batch's trees, built together (trees of at most 65,536 triangles
    that are still there, two or more of them) or alone: hits equal those of the scenes' own
    trees in both modes."""
    import torch

    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    ctx = cav.Context(0)
    data = [scenes.soup(n, seed=500 + k) for k, n in enumerate(sizes + [400])]
    dev = [(torch.from_numpy(p).cuda(), torch.from_numpy(i).cuda()) for p, i in data]
    batch = ctx.build_batch(dev, rounds=1)
    batch.pop().free()  # before any view was built
    rays = torch.from_numpy(scenes.closest_rays(3000, seed=7)).cuda()
    limit = torch.full((3000,), 0.6, device="cuda")
    for k, tree in enumerate(batch):
        single = ctx.build(*dev[k], rounds=1)
        for flags in (cav.TRACE_EXACT, cav.TRACE_FAST):
            for x, y in zip(tree.trace_closest(rays, flags=flags), single.trace_closest(rays, flags=flags)):
                assert torch.equal(x, y), (k, flags)
            assert torch.equal(tree.trace_any(rays, limit, flags=flags), single.trace_any(rays, limit, flags=flags))
        if k % 2:
            tree.free()
        single.free()
    ctx.sync_check()
