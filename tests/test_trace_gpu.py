"""Parity of the CUDA traversal (salty_trace) with the reference and the oracle.

The bar (closest hit): triangle ids bit-exact, ties to the lowest id; hit t within
1e-5 relative (the reference-compatible test in fact reproduces t bit for bit, which
is also asserted).  Any hit: occluded exactly when a closest hit exists.
"""
import os

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu

T_RTOL = 1e-5


def _scene(ctx, tris, **kw):
    import salty_gb300
    sc = ctx.upload_scene(tris, **kw)
    sc.build()
    return sc


def _check_closest(res, ids, t, exact_t=True):
    assert np.array_equal(res.ids, ids), f"{np.count_nonzero(res.ids != ids)} id mismatches of {ids.size}"
    hit = ids >= 0
    if hit.any():
        rel = np.abs(res.t[hit] - t[hit]) / np.abs(t[hit])
        assert rel.max() <= T_RTOL
        if exact_t:
            assert np.array_equal(res.t[hit], t[hit])
    assert np.all(np.isinf(res.t[~hit]))


def test_closest_hit_matches_reference_fixture_1m(gpu_soup_1m):
    import salty_gb300
    g = np.load(os.path.join(GOLDEN, "trace_soup_1m.npz"))
    rays = salty_gb300.microbench_rays(20260002, 65536, 1e-4)
    res = gpu_soup_1m.trace(rays)
    _check_closest(res, g["ids"], g["t"])


def test_closest_hit_matches_reference_fixture_30k(ctx):
    import salty_gb300
    g = np.load(os.path.join(GOLDEN, "trace_soup_30k.npz"))
    tris = salty_gb300.microbench_soup(int(g["soup_seed"]), int(g["n_tris"]))
    rays = salty_gb300.microbench_rays(int(g["ray_seed"]), int(g["n_rays"]), 1e-4)
    sc = _scene(ctx, tris)
    res = sc.trace(rays)
    _check_closest(res, g["ids"], g["t"])
    hit = g["ids"] >= 0
    assert np.array_equal(res.u[hit], g["u"][hit]) and np.array_equal(res.v[hit], g["v"][hit])


def test_full_workload_subset_matches_oracle(gpu_soup_1m, soup_1m, oracle, ctx):
    """All 16,777,216 microbenchmark rays on the device; a seeded random subset checked
    against the oracle, plus size-independent properties on every ray."""
    import torch
    import salty_gb300
    n = 16_777_216
    rays = salty_gb300.microbench_rays(20260002, n, 1e-4)
    d_rays = torch.from_numpy(rays).cuda()
    d_hits = torch.empty((n, 4), dtype=torch.float32, device="cuda")
    gpu_soup_1m.trace_raw(d_rays, d_hits)
    hits = d_hits.cpu().numpy()
    ids = hits[:, 1].view(np.int32)
    sub = np.random.default_rng(3).choice(n, 32768, replace=False)
    oid, ot, _, _ = oracle.trace(soup_1m, rays[sub], mode=0)
    assert np.array_equal(ids[sub], oid)
    h = oid >= 0
    assert np.array_equal(hits[sub, 0][h], ot[h])
    assert (ids >= 0).mean() > 0.97
    assert np.all((ids >= -1) & (ids < 1_000_000))
    # any hit: occluded iff a closest hit exists (every ray)
    d_any = torch.empty_like(d_hits)
    gpu_soup_1m.trace_raw(d_rays, d_any, any_hit=True)
    any_ids = d_any[:, 1].cpu().numpy().view(np.int32)
    assert np.array_equal(any_ids >= 0, ids >= 0)
    # the any-hit t is a real hit no nearer than the closest
    a_t = d_any[:, 0].cpu().numpy()
    hit = ids >= 0
    assert np.all(a_t[hit] >= hits[hit, 0])


def test_host_and_device_buffers_agree(gpu_soup_1m):
    import torch
    import salty_gb300
    rays = salty_gb300.microbench_rays(5, 3_000_001, 1e-4)  # spans two host chunks, ragged tail
    host = gpu_soup_1m.trace(rays)
    d_hits = torch.empty((rays.shape[0], 4), dtype=torch.float32, device="cuda")
    gpu_soup_1m.trace_raw(torch.from_numpy(rays).cuda(), d_hits)
    dev = d_hits.cpu().numpy()
    assert np.array_equal(host.ids, dev[:, 1].view(np.int32))
    assert np.array_equal(host.t, dev[:, 0])


@pytest.mark.parametrize("n", [0, 1, 31, 33, 1000])
def test_ragged_and_empty_ray_counts(ctx, oracle, n):
    import salty_gb300
    tris = salty_gb300.microbench_soup(21, 5000)
    sc = _scene(ctx, tris)
    rays = salty_gb300.microbench_rays(22, n, 1e-4)
    res = sc.trace(rays)
    assert res.ids.shape == (n,)
    if n:
        oid, ot, _, _ = oracle.trace(tris, rays, mode=0)
        _check_closest(res, oid, ot)


def test_single_triangle_and_axis_aligned_rays(ctx, oracle):
    tris = np.array([[0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0, 0.0]], np.float32)
    sc = _scene(ctx, tris)
    rays = np.array([
        [0.25, 0.25, -1.0, 1e-4, 0.0, 0.0, 1.0, np.inf],   # straight +z: hit at t = 1
        [0.25, 0.25, 1.0, 1e-4, 0.0, 0.0, -1.0, np.inf],   # straight -z: hit (two-sided)
        [0.25, 0.25, -1.0, 1e-4, 0.0, 0.0, -1.0, np.inf],  # away: miss
        [2.0, 2.0, -1.0, 1e-4, 0.0, 0.0, 1.0, np.inf],     # outside: miss
        [0.25, 0.25, -1.0, 1e-4, 0.0, 0.0, 1.0, 0.5],      # tmax before the triangle: miss
        [0.25, 0.25, -1.0, 2.0, 0.0, 0.0, 1.0, np.inf],    # tmin after the triangle: miss
        [-1.0, 0.25, 0.0, 1e-4, 1.0, 0.0, 0.0, np.inf],    # in the triangle's plane: miss
    ], np.float32)
    res = sc.trace(rays)
    oid, ot, _, _ = oracle.trace(tris, rays, mode=0)
    assert list(res.ids) == [0, 0, -1, -1, -1, -1, -1]
    _check_closest(res, oid, ot)
    assert res.t[0] == 1.0


def test_duplicate_triangles_tie_to_lowest_id(ctx, oracle):
    import salty_gb300
    base = salty_gb300.microbench_soup(51, 2000)
    tris = np.concatenate([base, base[::-1]])  # triangle i duplicated at 3999 - i
    sc = _scene(ctx, tris)
    rays = salty_gb300.microbench_rays(52, 20000, 1e-4)
    res = sc.trace(rays)
    oid, ot, _, _ = oracle.trace(tris, rays, mode=0)
    _check_closest(res, oid, ot)
    hit = res.ids >= 0
    assert hit.sum() > 100 and np.all(res.ids[hit] < 2000)


def test_degenerate_triangles_never_hit(ctx, oracle):
    import salty_gb300
    tris = salty_gb300.microbench_soup(61, 3000)
    tris[::3, 3:6] = tris[::3, 0:3]          # zero-area (repeated vertex)
    tris[1::7, 6:9] = 2 * tris[1::7, 3:6] - tris[1::7, 0:3]  # collinear
    sc = _scene(ctx, tris)
    rays = salty_gb300.microbench_rays(62, 20000, 1e-4)
    res = sc.trace(rays)
    oid, ot, _, _ = oracle.trace(tris, rays, mode=0)
    _check_closest(res, oid, ot)
    assert not np.any(np.isin(res.ids[res.ids >= 0], np.arange(0, 3000, 3)))


def test_watertight_mode_matches_oracle(ctx, oracle):
    import salty_gb300
    tris = salty_gb300.microbench_soup(71, 100000)
    sc = _scene(ctx, tris)
    rays = salty_gb300.microbench_rays(72, 20000, 1e-4)
    res = sc.trace(rays, watertight=True)
    oid, ot, _, _ = oracle.trace(tris, rays, mode=1)
    _check_closest(res, oid, ot, exact_t=False)


def test_watertight_closes_shared_edges(ctx):
    """A quad split along its diagonal: rays aimed at the diagonal hit in watertight mode;
    the reference test (strict inequalities) misses some of them."""
    quad = np.array([[0, 0, 0, 1, 0, 0, 1, 1, 0], [0, 0, 0, 1, 1, 0, 0, 1, 0]], np.float32)
    sc = _scene(ctx, quad)
    s = np.linspace(0.01, 0.99, 999, dtype=np.float32)
    rays = np.zeros((s.size, 8), np.float32)
    rays[:, 0] = s; rays[:, 1] = s; rays[:, 2] = -1.0; rays[:, 3] = 1e-4
    rays[:, 6] = 1.0; rays[:, 7] = np.inf
    wt = sc.trace(rays, watertight=True)
    assert np.all(wt.ids >= 0)


@pytest.mark.parametrize("bins,max_leaf", [(8, 1), (16, 2), (32, 3)])
def test_build_options_do_not_change_results(ctx, oracle, bins, max_leaf):
    import salty_gb300
    tris = salty_gb300.microbench_soup(81, 50000)
    sc = ctx.upload_scene(tris)
    info = sc.build(bins=bins, max_leaf=max_leaf)
    assert info["n_nodes"] > 0 and 0 < info["depth"] <= 40 and np.isfinite(info["sah_cost"])
    rays = salty_gb300.microbench_rays(82, 8192, 1e-4)
    res = sc.trace(rays)
    oid, ot, _, _ = oracle.trace(tris, rays, mode=0)
    _check_closest(res, oid, ot)


def test_counters_report_fetches(gpu_soup_1m):
    import salty_gb300
    rays = salty_gb300.microbench_rays(20260002, 100000, 1e-4)
    gpu_soup_1m.trace(rays, counters=True)
    st = gpu_soup_1m.last_stats
    assert st["node_fetches"] > st["rays"] and st["tri_fetches"] > 0


def test_errors_are_reported_not_crashing(ctx):
    import salty_gb300
    tris = salty_gb300.microbench_soup(91, 100)
    sc = ctx.upload_scene(tris)
    with pytest.raises(salty_gb300.SaltyError) as e:
        sc.trace(salty_gb300.microbench_rays(1, 10))
    assert e.value.status == salty_gb300.ERR_NOT_BUILT
    with pytest.raises(salty_gb300.SaltyError) as e:
        sc.build(bins=64)
    assert e.value.status == salty_gb300.ERR_INVALID_ARG
    with pytest.raises(salty_gb300.SaltyError):
        ctx.upload_scene(np.zeros((0, 9), np.float32))


def test_autotune_trace_keeps_results(ctx, gpu_soup_1m):
    """Every traversal launch shape gives the same hits; the autotuner picks one of them."""
    import torch
    import salty_gb300
    rays = torch.from_numpy(salty_gb300.microbench_rays(20260002, 1 << 20, 1e-4)).cuda()
    hits = torch.empty((1 << 20, 4), device="cuda")
    default = ctx.tuning
    gpu_soup_1m.trace_raw(rays, hits)
    ref = hits.cpu().numpy().view(np.int32).copy()
    t, ms = gpu_soup_1m.autotune_trace(rays)
    assert ms > 0 and t == ctx.tuning and t["trace_block"] in (64, 128, 256) and t["trace_regs"] in (56, 64)
    gpu_soup_1m.trace_raw(rays, hits)
    np.testing.assert_array_equal(hits.cpu().numpy().view(np.int32), ref)
    ctx.tuning = default


def _layout(kind, n):
    rng = np.random.default_rng(n)
    if kind == "soup":
        c = rng.random((n, 3))
    elif kind == "stacked":    # one centroid: no bin separates anything, halves by position
        c = np.full((n, 3), 0.5)
    else:                      # "chain": geometric spacing, each split peels off a few
        c = np.zeros((n, 3))
        c[:, 0] = 1.02 ** -np.arange(n)
    size = 0.02 if kind != "chain" else 0.01 * c[:, :1, None]
    return (c[:, None, :] + size * (rng.random((n, 3, 3)) - 0.5)).reshape(n, 9).astype(np.float32)


# Sizes around the builder's limits: one to a leaf (3), the 8- and 16-lane ranges, a block's
# subtree (512), a work item of the top levels (2048); every build must give the oracle's hits.
@pytest.mark.parametrize("kind", ["soup", "stacked", "chain"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 8, 9, 16, 17, 33, 512, 513, 2049, 5000])
@pytest.mark.parametrize("bins,max_leaf", [(32, 3), (8, 1)])
def test_build_at_size_limits(ctx, oracle, kind, n, bins, max_leaf):
    tris = _layout(kind, min(n, 2049) if kind == "chain" else n)
    n = tris.shape[0]
    rng = np.random.default_rng(5)
    org = rng.uniform(-1, 2, (512, 3))
    to = tris.reshape(-1, 3, 3).mean(1)[rng.integers(0, n, 512)] + rng.normal(0, 0.003, (512, 3))
    rays = np.zeros((512, 8), np.float32)
    rays[:, :3], rays[:, 4:7] = org, (to - org) / np.linalg.norm(to - org, axis=1, keepdims=True)
    rays[:, 3], rays[:, 7] = 1e-4, np.inf
    s = ctx.upload_scene(tris)
    info = s.build(bins=bins, max_leaf=max_leaf)
    assert info["n_binary"] <= 2 * n - 1 and info["n_nodes"] >= 1
    res = s.trace(rays)
    oid, ot, _, _ = oracle.trace(tris, rays, mode=0)
    np.testing.assert_array_equal(res.ids, oid)
    np.testing.assert_array_equal(res.t[oid >= 0], ot[oid >= 0])
    s.close()


# The queueing walk (postpone 1) against the walk in which lanes test their own triangles
# (postpone 2), bit for bit: ray counts around a warp, its least share of rays and its refill
# size; leaf-heavy and empty regions; the rays' own limits.
@pytest.mark.parametrize("n", [1, 5, 6, 31, 33, 700, 40000])
@pytest.mark.parametrize("watertight", [False, True])
def test_queueing_walk_matches_own_tests(ctx, n, watertight):
    import salty_gb300
    tris = salty_gb300.microbench_soup(17, 40000)
    tris[:500] = tris[0]                      # equal distances
    sc = _scene(ctx, tris)
    assert sc.info["depth"] > 3
    rays = salty_gb300.microbench_rays(n, n, 1e-4)
    rays[::3, 7] = 2.0                        # tmax among the hits
    rays[1::5, 3] = 1.9                       # tmin too
    if n > 30:
        rays[7, 7] = -1.0                     # nothing can be hit
        rays[8, 7] = np.nan                   # bounds nothing
        rays[9, 3] = -5.0                     # taken as 0
        rays[10, 4:7] = (0.0, 0.0, 1.0)
    base = ctx.tuning
    try:
        got, occ = {}, {}
        for post in (1, 2):
            ctx.tuning = {"trace_postpone": post}
            got[post] = sc.trace(rays, watertight=watertight)
            occ[post] = sc.trace(rays, any_hit=True, watertight=watertight).ids >= 0
    finally:
        ctx.tuning = base
    for f in ("ids", "t", "u", "v"):
        np.testing.assert_array_equal(getattr(got[1], f), getattr(got[2], f))
    np.testing.assert_array_equal(occ[1], got[1].ids >= 0)
    np.testing.assert_array_equal(occ[1], occ[2])
    sc.close()


# More rays than lanes in a tree of eight levels or more take the queueing walk under either
# test; one lane's worth past the line and a ragged larger size, bit for bit as above.
@pytest.mark.parametrize("extra", [1, 44353])
@pytest.mark.parametrize("watertight", [False, True])
def test_queueing_walk_on_deep_trees(ctx, extra, watertight):
    import salty_gb300
    import torch
    tris = salty_gb300.microbench_soup(17, 300000)
    tris[:500] = tris[0]
    sc = _scene(ctx, tris)
    assert sc.info["depth"] >= 8
    n = 1024 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    rays = salty_gb300.microbench_rays(5, n, 1e-4)
    rays[::3, 7] = 2.0
    rays[1::5, 3] = 1.9
    rays[7, 7] = -1.0
    rays[8, 7] = np.nan
    rays[9, 3] = -5.0
    rays[10, 4:7] = (0.0, 0.0, 1.0)
    base = ctx.tuning
    try:
        got, occ = {}, {}
        for post in (1, 2):
            ctx.tuning = {"trace_postpone": post}
            got[post] = sc.trace(rays, watertight=watertight)
            occ[post] = sc.trace(rays, any_hit=True, watertight=watertight).ids >= 0
    finally:
        ctx.tuning = base
    for f in ("ids", "t", "u", "v"):
        np.testing.assert_array_equal(getattr(got[1], f), getattr(got[2], f))
    np.testing.assert_array_equal(occ[1], got[1].ids >= 0)
    np.testing.assert_array_equal(occ[1], occ[2])
    sc.close()


# Host arrays in one chunk, two, and two with a ragged second one: the same hits as from device
# memory.
@pytest.mark.parametrize("n", [1 << 18, (1 << 18) + 1, (1 << 19) + 3])
def test_host_chunks_match_device_arrays(ctx, n):
    import salty_gb300
    import torch
    sc = _scene(ctx, salty_gb300.microbench_soup(3, 2000))
    rays = salty_gb300.microbench_rays(4, n, 1e-4)
    host = np.full((n, 4), -7.0, np.float32)
    sc.trace_raw(rays, host)
    dev = torch.empty((n, 4), device="cuda")
    sc.trace_raw(torch.from_numpy(rays).cuda(), dev)
    np.testing.assert_array_equal(host.view(np.uint32), dev.cpu().numpy().view(np.uint32))
    sc.close()


def _doubled_soup(n, seed):
    """Every triangle twice, the ids shuffled."""
    import salty_gb300
    t = salty_gb300.microbench_soup(seed, n)
    return np.ascontiguousarray(np.concatenate([t, t])[np.random.default_rng(seed).permutation(2 * n)])


# Coincident triangles: the lowest id wins under either test, whichever of the two a walk
# tests first (the queueing walk's order depends on the rays that share a warp), so calls repeat
# bit for bit.  More rays than lanes, so that the deep trees take the queueing walk.
@pytest.mark.parametrize("n", [3000, 100000])
@pytest.mark.parametrize("watertight", [False, True])
def test_coincident_triangles_give_the_lowest_id(ctx, oracle, n, watertight):
    import salty_gb300
    import torch
    tris = _doubled_soup(n, 23)
    sc = _scene(ctx, tris)
    assert n < 100000 or sc.info["depth"] >= 7
    rays = salty_gb300.microbench_rays(6, 1024 * torch.cuda.get_device_properties(0).multi_processor_count + 77, 1e-4)
    res = [sc.trace(rays, watertight=watertight) for _ in range(3)]
    oid, ot, _, _ = oracle.trace(tris, rays, mode=1 if watertight else 0)
    for r in res:
        np.testing.assert_array_equal(r.ids, oid)
        np.testing.assert_array_equal(r.t[oid >= 0], ot[oid >= 0])
        np.testing.assert_array_equal(r.u, res[0].u)
        np.testing.assert_array_equal(r.v, res[0].v)
    sc.close()


# A watertight hit at its ray's own limit: kept when both T / det as the oracle compares it and
# the rounded t are within the limit; limits at the hit distances and one unit in the last
# place either side.
@pytest.mark.parametrize("step", [-1, 0, 1])
def test_watertight_hits_at_the_ray_limit(ctx, oracle, step):
    import salty_gb300
    tris = _doubled_soup(20000, 29)
    sc = _scene(ctx, tris)
    rays = salty_gb300.microbench_rays(8, 40000, 1e-4)
    _, ot, _, _ = oracle.trace(tris, rays, mode=1)
    rays[:, 7] = np.where(np.isinf(ot), ot, (ot.view(np.int32) + step).view(np.float32))
    oid, ot, _, _ = oracle.trace(tris, rays, mode=1)
    res = sc.trace(rays, watertight=True)
    np.testing.assert_array_equal(res.ids, np.where(ot <= rays[:, 7], oid, -1))
    sc.close()


def _whole_and_pieces(sc, rays, **kw):
    """The same rays in one call and in calls of no more rays than lanes: the deep trees'
    queueing walk, and the walk in which lanes test their own triangles."""
    import torch
    lanes = 1024 * torch.cuda.get_device_properties(0).multi_processor_count
    assert len(rays) > lanes
    whole = sc.trace(rays, **kw)
    parts = [sc.trace(rays[k:k + lanes], **kw) for k in range(0, len(rays), lanes)]
    bits = lambda r: np.stack([r.t.view(np.int32), r.ids, r.u.view(np.int32), r.v.view(np.int32)], 1)
    return bits(whole), np.concatenate([bits(p) for p in parts])


# Any hit returns one and the same hit of a ray, the first of its walk, in either walk and in
# every call, among coincident triangles too.
@pytest.mark.parametrize("watertight", [False, True])
def test_any_hit_is_the_same_hit_in_every_call(ctx, watertight):
    import salty_gb300
    sc = _scene(ctx, _doubled_soup(400000, 31))
    assert sc.info["depth"] >= (7 if watertight else 8)
    rays = salty_gb300.microbench_rays(9, 300001, 1e-4)
    rays[::3, 7] = 2.0
    for _ in range(2):
        whole, pieces = _whole_and_pieces(sc, rays, any_hit=True, watertight=watertight)
        np.testing.assert_array_equal(whole, pieces)
    sc.close()


# Rays from points on the triangles themselves: distances of 0, of either sign, and a few
# 1e-7, in both walks and under both tests.
@pytest.mark.parametrize("watertight", [False, True])
def test_rays_leaving_surfaces(ctx, watertight):
    import salty_gb300
    tris = salty_gb300.microbench_soup(37, 300000)
    sc = _scene(ctx, tris)
    assert sc.info["depth"] >= 8
    rng = np.random.default_rng(3)
    n = 1 << 20
    w = rng.dirichlet((1, 1, 1), n).astype(np.float32)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = (tris.reshape(-1, 3, 3)[rng.integers(0, len(tris), n)] * w[:, :, None]).sum(1)
    d = rng.normal(size=(n, 3))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = np.inf
    whole, pieces = _whole_and_pieces(sc, rays, watertight=watertight)
    assert np.count_nonzero(pieces[:, 0] == np.float32(-0.0).view(np.int32)) > 50
    np.testing.assert_array_equal(whole, pieces)
    sc.close()


# A scene built once leaves no build workspace behind; one built again keeps a bounded one,
# which goes with the scene.  (Sizes to the driver's 2 MB blocks.)
def test_build_workspace_is_given_back(salty_lib):
    import salty_gb300
    import torch
    free = lambda: torch.cuda.mem_get_info()[0]
    n, slack = 1000000, 8 << 20
    tris = salty_gb300.microbench_soup(41, n)
    with salty_gb300.Context(0) as c:
        w = c.upload_scene(tris[:1000])
        w.build()                              # loads the kernels
        w.close()
        before = free()
        s = c.upload_scene(tris)
        uploaded = free()
        s.build()
        tree = uploaded - free()
        assert tree <= (n + 1) * 80 + n * 48 + slack
        s.build()
        kept = uploaded - free() - tree
        assert kept <= (512 << 20) + slack
        other = c.upload_scene(tris[:2000])
        other.build()
        other.close()
        s.close()
        assert before - free() <= slack


# A box of 2^-60 in a node of 2^100: its upper plane is an index of one, not of zero, so a ray
# that starts inside meets what is there.
@pytest.mark.parametrize("watertight", [False, True])
def test_tiny_boxes_in_huge_nodes(ctx, watertight):
    tris = np.zeros((20, 3, 3), np.float32)
    tris[:, 0, 1:], tris[:, 1, 1:], tris[:, 2, 1:] = (0.0, 0.0), (0.8, 0.0), (0.0, 0.8)
    tris[:, :, 1] += np.arange(20, dtype=np.float32)[:, None]
    tris[:16:2, :, 0] = 2.0 ** -60
    tris[16:, :, 0] = 2.0 ** 100
    sc = _scene(ctx, tris.reshape(-1, 9))
    near = np.arange(0, 16, 2)
    rays = np.zeros((len(near), 8), np.float32)
    rays[:, 0], rays[:, 1], rays[:, 2] = 2.0 ** -61, near + 0.2, 0.2
    rays[:, 4], rays[:, 7] = 1.0, np.inf
    res = sc.trace(rays, watertight=watertight)
    np.testing.assert_array_equal(res.ids, near)
    np.testing.assert_array_equal(res.t, np.full(len(near), 2.0 ** -61, np.float32))
    sc.close()


# Pinned arrays of more than 2^18 rays go in halves in trees of six levels; pageable ones, whose
# copies overlap nothing, and those of which one stays on the device go whole.  The hits are the same.
@pytest.mark.parametrize("n", [1 << 18, (1 << 19) + 3])
def test_chunks_of_pinned_and_pageable_arrays(ctx, n):
    import salty_gb300
    import torch
    sc = _scene(ctx, salty_gb300.microbench_soup(3, 30000))
    assert sc.info["depth"] == 6
    rays = salty_gb300.microbench_rays(4, n, 1e-4)
    pinned_rays, pinned_hits, dev_hits = ctx.pinned((n, 8)), ctx.pinned((n, 4)), torch.empty((n, 4), device="cuda")
    pinned_rays[:] = rays
    pageable = lambda: np.empty((n, 4), np.float32)
    hits = {}
    for name, r, h in (("pageable", rays, pageable()), ("pinned", pinned_rays, pinned_hits),
                       ("rays pinned", pinned_rays, pageable()), ("to the device", pinned_rays, dev_hits)):
        st = sc.trace_raw(r, h)
        assert st["launches"] == (2 if name == "pinned" and n > 1 << 18 else 1), name
        hits[name] = (h.cpu().numpy() if h is dev_hits else h).view(np.uint32).copy()
    for name in hits:
        np.testing.assert_array_equal(hits[name], hits["pageable"])
    sc.close()
