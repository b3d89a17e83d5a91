"""GPU parity of the CUDA path (through the C ABI) against the reference.

* Golden fixtures (tests/golden/*.npz, produced by the reference's own CUDA code):
  Morton codes, sort order, the node array after N treelet rounds and closest/any-hit
  results must be bit-identical.
* The live reference build (oracle/_ref/libcavref.so, when present) at the full 1M
  triangle size of the soup workload: same bit-exact checks.
* The C oracle at medium sizes, fed the GPU's Morton codes, for the integer and
  treelet stages (exact) and traversal (ids equal except near-ties).
"""
import numpy as np
import pytest

from conftest import golden_files, lbvh_matches_reference, load_golden, nodes_equal

pytestmark = pytest.mark.gpu

GOLDEN = golden_files()


def _cuda(a, dtype=None):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda() if dtype is None else torch.from_numpy(
        np.ascontiguousarray(a, dtype)).cuda()


def _build(ctx, pos, idx, mesh=None, rounds=0, bounds=None):
    return ctx.build(_cuda(pos, np.float32), _cuda(idx, np.int32), None if mesh is None else _cuda(mesh, np.int32),
                     scene_bounds=bounds, rounds=int(rounds))


@pytest.mark.parametrize("path", GOLDEN, ids=[p.stem for p in GOLDEN])
def test_golden_lbvh_matches_reference(cuda_ctx, path):
    """Morton codes, sort order and topology bit-exact against the reference's own LBVH;
    boxes bit-exact except where the reference's unfenced refit raced (explained node by node)."""
    g = load_golden(path)
    bvh = _build(cuda_ctx, g["pos"], g["idx"], g["mesh_ids"], 0)
    mu, ms, pr = bvh.export_stages()
    assert np.array_equal(mu, g["codes"]), f"Morton codes differ at {np.nonzero(mu != g['codes'])[0][:10]}"
    assert np.array_equal(ms, g["sorted"])
    assert np.array_equal(pr, g["perm"])
    nodes = bvh.export_nodes()
    lbvh_matches_reference(nodes, g["merged_ref"], g["merged"], path.stem)
    nodes_equal(nodes, g["merged"], path.stem)
    cuda_ctx.sync_check()
    bvh.free()


@pytest.mark.parametrize("path", GOLDEN, ids=[p.stem for p in GOLDEN])
def test_golden_treelet_rounds(cuda_ctx, path):
    """3 treelet rounds on the same LBVH: bit-exact against the oracle restatement."""
    g = load_golden(path)
    bvh = _build(cuda_ctx, g["pos"], g["idx"], g["mesh_ids"], 3)
    nodes_equal(bvh.export_nodes(), g["final3"], path.stem)
    cuda_ctx.sync_check()
    bvh.free()


@pytest.mark.parametrize("rounds", [0, 3])
@pytest.mark.parametrize("path", GOLDEN, ids=[p.stem for p in GOLDEN])
def test_golden_trace_bit_exact(cuda_ctx, path, rounds):
    """Closest/any hit bit-exact against the reference's verbatim traversal on the same tree."""
    import cavalry_b200 as cav

    g = load_golden(path)
    cp, ct, so = (g["c_prim"], g["c_t"], g["s_occ"]) if rounds == 0 else (g["c3_prim"], g["c3_t"], g["s3_occ"])
    if (cp == -3).all():
        pytest.skip("tree deeper than the reference's fixed traversal stack; no reference results")
    bvh = _build(cuda_ctx, g["pos"], g["idx"], g["mesh_ids"], rounds)
    prim, t, uv = bvh.trace_closest(_cuda(g["rays"]))
    prim = prim.cpu().numpy()
    t = t.cpu().numpy()
    assert np.array_equal(prim, cp), f"closest ids differ at {np.nonzero(prim != cp)[0][:10]}"
    hit = prim >= 0
    assert np.array_equal(t[hit].view(np.uint32), ct[hit].view(np.uint32))
    occ = bvh.trace_any(_cuda(g["srays"]), _cuda(g["s_limit"]), _cuda(g["s_excl"])).cpu().numpy()
    assert np.array_equal(occ, so), f"any-hit differs at {np.nonzero(occ != so)[0][:10]}"
    # culling on pop may only change which of exactly-equal-t hits is reported
    p2, t2, _ = bvh.trace_closest(_cuda(g["rays"]), flags=cav.TRACE_CULL_ON_POP)
    p2 = p2.cpu().numpy()
    t2 = t2.cpu().numpy()
    assert np.array_equal(p2 >= 0, hit)
    assert np.array_equal(t2[hit].view(np.uint32), t[hit].view(np.uint32))
    o2 = bvh.trace_any(_cuda(g["srays"]), _cuda(g["s_limit"]), _cuda(g["s_excl"]), flags=cav.TRACE_CULL_ON_POP)
    assert np.array_equal(o2.cpu().numpy(), occ)
    cuda_ctx.sync_check()
    bvh.free()


@pytest.mark.parametrize("path", GOLDEN[:3], ids=[p.stem for p in GOLDEN[:3]])
def test_host_buffer_path_matches_device_path(cuda_ctx, path):
    g = load_golden(path)
    bvh = _build(cuda_ctx, g["pos"], g["idx"], g["mesh_ids"], 0)
    prim_h, t_h, uv_h = bvh.trace_closest_host(np.ascontiguousarray(g["rays"]))
    assert np.array_equal(prim_h, g["c_prim"])
    occ_h = bvh.trace_any_host(np.ascontiguousarray(g["srays"]), np.ascontiguousarray(g["s_limit"]),
                               np.ascontiguousarray(g["s_excl"]))
    assert np.array_equal(occ_h, g["s_occ"])
    bvh.free()


def _ref_or_skip():
    from oracle import pyoracle as po

    if not po.ref_available():
        pytest.skip("oracle/_ref/libcavref.so not built (reference sources absent when building)")
    return po


def test_live_reference_soup_1m(cuda_ctx):
    """Full-size soup workload (1M triangles) against the reference's own code on the GPU:
    LBVH stages (bit-exact; boxes race-aware), then the reference's verbatim traversal on
    our 3-round tree must give bit-identical closest and any hits for 1M rays each."""
    po = _ref_or_skip()
    from cavalry_b200 import scenes
    from conftest import lbvh_matches_reference

    pos, idx = scenes.soup(1_000_000, seed=2)
    ref = po.RefScene(pos, idx, rounds=0, id_mode=1, dump=True)
    bvh0 = _build(cuda_ctx, pos, idx, rounds=0)
    mu, ms, pr = bvh0.export_stages()
    assert np.array_equal(mu, ref.codes)
    assert np.array_equal(ms, ref.sorted)
    assert np.array_equal(pr, ref.perm)
    o = po.build(pos, idx, codes=ref.codes, rounds=0)
    sites = lbvh_matches_reference(bvh0.export_nodes(), ref.merged, o["merged"], "soup1m")
    print(f"reference refit race sites at 1M: {sites}")
    bvh0.free()
    bvh = _build(cuda_ctx, pos, idx, rounds=3)
    ref.load_nodes(bvh.export_nodes())
    assert ref.depth <= 62, f"tree too deep for the reference's fixed stack ({ref.depth})"
    rays = scenes.closest_rays(1 << 20, seed=20)
    prim, t, _ = bvh.trace_closest(_cuda(rays))
    rp, rt, _ = ref.trace_closest(rays)
    prim = prim.cpu().numpy()
    assert np.array_equal(prim, rp), f"{(prim != rp).sum()} closest ids differ"
    hit = prim >= 0
    assert np.array_equal(t.cpu().numpy()[hit].view(np.uint32), rt[hit].view(np.uint32))
    srays, lim = scenes.shadow_rays(1 << 20, seed=21)
    occ = bvh.trace_any(_cuda(srays), _cuda(lim)).cpu().numpy()
    ro, _ = ref.trace_any(srays, lim)
    assert np.array_equal(occ, ro)
    ref.free()
    bvh.free()


@pytest.mark.parametrize("n,rounds,seed", [(34, 2, 0), (1000, 3, 11), (4097, 2, 13), (100_000, 3, 31)])
def test_treelet_rounds_match_oracle(cuda_ctx, n, rounds, seed):
    """Treelet rounds (not runnable in the reference on this GPU) against the oracle restatement."""
    from cavalry_b200 import scenes
    from oracle import pyoracle as po

    if n == 34:
        room = scenes.mini_room()
        pos, idx = room["positions"], room["indices"][:34]
    else:
        pos, idx = scenes.soup(n, seed=seed)
    bvh = _build(cuda_ctx, pos, idx, rounds=rounds)
    mu, _, _ = bvh.export_stages()
    o = po.build(pos, idx, codes=mu, rounds=rounds)
    nodes_equal(bvh.export_nodes(), o["final"], f"treelet n={n} r={rounds}")
    cuda_ctx.sync_check()
    bvh.free()


def test_oracle_integer_and_treelet_stages_exact_100k(cuda_ctx):
    """The C oracle fed the GPU's Morton codes reproduces sort, radix tree, refit and 3 treelet rounds exactly."""
    from cavalry_b200 import scenes
    from oracle import pyoracle as po

    pos, idx = scenes.soup(100_000, seed=31)
    bvh = _build(cuda_ctx, pos, idx, rounds=3)
    mu, ms, pr = bvh.export_stages()
    o = po.build(pos, idx, codes=mu, rounds=3)
    assert np.array_equal(ms, o["sorted"])
    assert np.array_equal(pr, o["perm"])
    nodes_equal(bvh.export_nodes(), o["final"], "oracle_100k")
    # Morton codes from the oracle's IEEE division: equal up to one cell on an axis
    from test_oracle_golden import morton_close

    morton_close(mu, po.morton(pos, idx, o["bounds"]))
    bvh.free()


def test_trace_matches_oracle_except_ties(cuda_ctx):
    from cavalry_b200 import scenes
    from oracle import pyoracle as po

    pos, idx = scenes.soup(50_000, seed=32)
    bvh = _build(cuda_ctx, pos, idx, rounds=2)
    mu, _, _ = bvh.export_stages()
    o = po.build(pos, idx, codes=mu, rounds=2)
    rays = scenes.closest_rays(200_000, seed=33)
    prim, t, _ = bvh.trace_closest(_cuda(rays))
    prim = prim.cpu().numpy()
    t = t.cpu().numpy()
    op, ot, _, _ = po.trace_closest(o["final"], pos, idx, rays)
    same = prim == op
    assert same.mean() > 0.9999, f"{(~same).sum()} of {len(prim)} ids differ"
    both = (prim >= 0) & same
    rel = np.abs(t[both] - ot[both]) / np.maximum(np.abs(ot[both]), 1e-30)
    assert rel.max() <= 1e-6 * 4, rel.max()
    bvh.free()


def test_full_size_properties_soup_1m(cuda_ctx):
    """Size-independent properties at the full workload: 1M triangles, 4M closest + 4M any-hit rays."""
    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    pos, idx = scenes.soup(1_000_000, seed=2)
    bvh = _build(cuda_ctx, pos, idx, rounds=3)
    nodes = bvh.export_nodes()
    leaf = nodes["is_leaf"].astype(bool)
    assert leaf.sum() == 1_000_000
    assert np.array_equal(np.sort(nodes["prim_begin"][leaf]), np.arange(1_000_000))
    inner = np.nonzero(~leaf)[0]
    for side in ("left", "right"):
        ch = nodes[side][inner]
        assert (nodes["bmin"][ch] >= nodes["bmin"][inner]).all()
        assert (nodes["bmax"][ch] <= nodes["bmax"][inner]).all()
    children = np.concatenate([nodes["left"][inner], nodes["right"][inner]])
    assert np.array_equal(np.sort(children), np.arange(1, 2 * 1_000_000 - 1))
    rays = _cuda(scenes.closest_rays(4 << 20, seed=20))
    p0, t0, _ = bvh.trace_closest(rays)
    p1, t1, _ = bvh.trace_closest(rays, flags=cav.TRACE_CULL_ON_POP)
    assert bool(((p0 >= 0) == (p1 >= 0)).all())
    hit = p0 >= 0
    assert bool((t0[hit] == t1[hit]).all())
    srays, lim = scenes.shadow_rays(4 << 20, seed=21)
    occ = bvh.trace_any(_cuda(srays), _cuda(lim)).cpu().numpy()
    pc, tc, _ = bvh.trace_closest(_cuda(srays))
    closer = ((pc.cpu().numpy() >= 0) & (tc.cpu().numpy() < lim)).astype(np.uint8)
    assert (occ != closer).mean() < 1e-5
    cuda_ctx.sync_check()
    bvh.free()


def test_build_is_deterministic_and_stream_ordered(cuda_ctx):
    import torch
    from cavalry_b200 import scenes

    pos, idx = scenes.soup(200_000, seed=41)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        a = cuda_ctx.build(_cuda(pos), _cuda(idx), rounds=3, stream=s)
        na = a.export_nodes(stream=s)
    b = _build(cuda_ctx, pos, idx, rounds=3)
    nodes_equal(na, b.export_nodes(), "determinism")
    a.free()
    b.free()


def test_deep_tree_traversal_matches_oracle(cuda_ctx):
    """300 identical triangles: 3 treelet rounds give a tree deeper than the reference's
    64-entry stack.  The reference would write past its stack; ours (128 entries, checked)
    must still agree with the oracle."""
    from oracle import pyoracle as po

    path = [p for p in GOLDEN if p.stem == "dup300"]
    if not path:
        pytest.skip("fixture missing")
    g = load_golden(path[0])
    bvh = _build(cuda_ctx, g["pos"], g["idx"], g["mesh_ids"], 3)
    assert bvh.depth() > 62
    prim, t, _ = bvh.trace_closest(_cuda(g["rays"]))
    op, ot, _, _ = po.trace_closest(g["final3"], g["pos"], g["idx"], g["rays"])
    prim = prim.cpu().numpy()
    assert (prim != -2).all()
    hit = prim >= 0
    assert np.array_equal(hit, op >= 0)
    assert np.allclose(t.cpu().numpy()[hit], ot[hit], rtol=4e-6)
    cuda_ctx.sync_check()
    bvh.free()


def test_invalid_arguments_are_reported(cuda_ctx):
    import torch

    import cavalry_b200 as cav

    pos = torch.zeros((3, 3), dtype=torch.float32, device="cuda")
    idx = torch.zeros((1, 3), dtype=torch.int32, device="cuda")
    with pytest.raises(cav.CavError):
        cuda_ctx.build(pos, idx, rounds=0)  # a single triangle is below the minimum of 2
    with pytest.raises(cav.CavError):
        cuda_ctx.set_trace_config(block_threads=33)


def test_host_buffer_path_over_several_chunks(cuda_ctx):
    """The host-buffer entry points pipeline chunks of 4M rays over two streams.  4,195,304
    rays make two chunks, the second ragged; with pageable (numpy) and with pinned (torch)
    buffers, closest and any hit equal the device path's results."""
    import torch

    from cavalry_b200 import scenes

    pos, idx = scenes.soup(20_000, seed=61)
    bvh = cuda_ctx.build(torch.from_numpy(pos).cuda(), torch.from_numpy(idx).cuda(), rounds=2)
    n = (1 << 22) + 1000
    rays = scenes.closest_rays(n, seed=62)
    srays, lim = scenes.shadow_rays(n, seed=63)
    prim_d, t_d, uv_d = (a.cpu().numpy() for a in bvh.trace_closest(torch.from_numpy(rays).cuda()))
    occ_d = bvh.trace_any(torch.from_numpy(srays).cuda(), torch.from_numpy(lim).cuda()).cpu().numpy()
    prim_h, t_h, uv_h = bvh.trace_closest_host(rays)
    occ_h = bvh.trace_any_host(srays, lim)
    assert np.array_equal(prim_h, prim_d) and np.array_equal(t_h.view(np.uint32), t_d.view(np.uint32))
    assert np.array_equal(uv_h.view(np.uint32), uv_d.view(np.uint32)) and np.array_equal(occ_h, occ_d)
    h_rays = torch.from_numpy(rays).pin_memory()
    out = (torch.empty(n, dtype=torch.int32).pin_memory(), torch.empty(n, dtype=torch.float32).pin_memory(),
           torch.empty((n, 2), dtype=torch.float32).pin_memory())
    bvh.trace_closest_host(h_rays, out=out)
    occ_p = torch.empty(n, dtype=torch.uint8).pin_memory()
    bvh.trace_any_host(torch.from_numpy(srays).pin_memory(), torch.from_numpy(lim).pin_memory(), out=occ_p)
    cuda_ctx.sync_check()
    assert np.array_equal(out[0].numpy(), prim_d) and np.array_equal(out[1].numpy().view(np.uint32), t_d.view(np.uint32))
    assert np.array_equal(occ_p.numpy(), occ_d)
    bvh.free()


@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19, 3 * (1 << 18) + 1, (1 << 20) + 3])
def test_host_buffer_path_in_parts(cuda_ctx, n):
    """Any-hit calls and calls with pageable buffers are cut into up to four chunks of 2^18
    rays or more (the last one ragged): one, two, three and four of them."""
    import torch

    from cavalry_b200 import scenes

    pos, idx = scenes.soup(3000, seed=64)
    bvh = cuda_ctx.build(torch.from_numpy(pos).cuda(), torch.from_numpy(idx).cuda())
    rays = scenes.closest_rays(n, seed=65)
    srays, lim = scenes.shadow_rays(n, seed=66)
    want = [a.cpu().numpy() for a in bvh.trace_closest(torch.from_numpy(rays).cuda())]
    occ = bvh.trace_any(torch.from_numpy(srays).cuda(), torch.from_numpy(lim).cuda()).cpu().numpy()
    for a, b in zip(bvh.trace_closest_host(rays), want):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert np.array_equal(bvh.trace_any_host(srays, lim), occ)
    out = torch.full((n,), 9, dtype=torch.uint8).pin_memory()
    bvh.trace_any_host(torch.from_numpy(srays).pin_memory(), torch.from_numpy(lim).pin_memory(), out=out)
    assert np.array_equal(out.numpy(), occ)
    bvh.free()


@pytest.mark.parametrize("n", [7, 8, 50, 1000, 5000])
@pytest.mark.parametrize("rounds", [1, 3])
def test_treelets_on_ties_match_oracle(cuda_ctx, n, rounds):
    """Vertices on a small integer lattice: areas are exact, so partitions tie everywhere and the
    choice among equal costs (in every subset size) decides the tree."""
    import torch

    from oracle import pyoracle as po

    rng = np.random.default_rng(n + rounds)
    pos = rng.integers(0, 9, (3 * n, 3)).astype(np.float32)
    pos[::5] = pos[0]
    idx = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    bvh = cuda_ctx.build(torch.from_numpy(pos).cuda(), torch.from_numpy(idx).cuda(), rounds=rounds)
    mu, ms, perm = bvh.export_stages()
    o = po.build(pos, idx, codes=mu, rounds=rounds)
    assert np.array_equal(ms, o["sorted"]) and np.array_equal(perm, o["perm"])
    nodes_equal(bvh.export_nodes(), o["final"], f"lattice {n} rounds {rounds}")
    cuda_ctx.sync_check()
    bvh.free()


@pytest.mark.parametrize("level,rounds", [(1, 1), (2, 3), (3, 3)])
def test_treelets_on_icospheres_match_oracle(cuda_ctx, level, rounds):
    """Icospheres' triangles come in near-equal pairs, whose partitions' costs are a rounding apart:
    the trees are the oracle's bit for bit with the treelet pass's own contraction of surface
    areas; with the build's contraction (the oracle's default) 0.4, 5.6 and 10 % of the nodes
    differ in these scenes."""
    import torch

    from cavalry_b200 import scenes
    from oracle import pyoracle as po

    s = scenes.sphere_scene(8, level, seed=5)
    pos, idx = s["positions"], s["indices"]
    bvh = cuda_ctx.build(torch.from_numpy(pos).cuda(), torch.from_numpy(idx).cuda(), rounds=rounds)
    mu, _, _ = bvh.export_stages()
    got = bvh.export_nodes()
    o = po.build(pos, idx, codes=mu, rounds=rounds, other_area=True)
    nodes_equal(got, o["final"], f"icospheres level {level} rounds {rounds}")
    o = po.build(pos, idx, codes=mu, rounds=rounds)["final"]
    same = (got["left"] == o["left"]) & (got["right"] == o["right"]) & (got["bmin"] == o["bmin"]).all(1)
    same &= (got["bmax"] == o["bmax"]).all(1)
    print(f"level {level} rounds {rounds}: {1 - same.mean():.4f} of the nodes differ")
    assert 0.85 < same.mean() < 1.0
    bvh.free()
