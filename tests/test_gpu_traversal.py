"""Closest-hit / any-hit parity of the CUDA traversal.

* On the reference's own tree, ids, t, u, v are bit-exact to the golden
  vectors produced by executing the reference's bvh_intersect.
* On the LBVH, the closest-hit triangle id is bit-exact to the oracle except
  for rays within 1e-6 (barycentric) of a triangle edge and exact t ties;
  both are excluded and counted, and every excluded mismatch is verified to
  be an equally close hit.  t, u, v agree to 1e-5 relative (they are
  bit-exact for the same triangle).
"""
import os

import numpy as np
import pytest

import golden_scenes as gs
import roxy_native as nat
from oracle import oracle, parity

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")


def _scene(v0, v1, v2, method, leaf):
    sc = nat.NativeScene()
    sc.set_triangles(v0, v1, v2)
    sc.set_materials([0], [[0.5, 0.5, 0.5]], [0.0], [1.0], [0.0])
    sc.build_bvh(method, leaf, True)
    return sc


def test_reference_tree_bit_exact_against_reference_traversal():
    g = np.load(os.path.join(GOLD, "traversal.npz"))
    for case in g["case_names"]:
        c = {k.split("/", 1)[1]: g[k] for k in g.files if k.startswith(f"{case}/")}
        sc = _scene(c["v0"], c["v1"], c["v2"], nat.RX_BVH_REFERENCE, int(c["leaf"]))
        t, idx, u, v = sc.trace_closest(c["ro"], c["rd"])
        ref_idx = np.where(c["idx"] >= 0, c["order"][np.maximum(c["idx"], 0)], -1)
        np.testing.assert_array_equal(idx, ref_idx, err_msg=case)
        hit = idx >= 0
        assert np.array_equal(t[hit].view(np.uint32), c["t"][hit].view(np.uint32))
        assert np.array_equal(u[hit].view(np.uint32), c["u"][hit].view(np.uint32))
        assert np.array_equal(v[hit].view(np.uint32), c["v"][hit].view(np.uint32))
        occ = sc.trace_any(c["ro"], c["rd"], c["max_t"])
        np.testing.assert_array_equal(occ, c["occluded"], err_msg=case)


def _parity(v0, v1, v2, ro, rd, method=nat.RX_BVH_LBVH_SAH, leaf=4):
    bvh = oracle.bvh_build_morton(v0, v1, v2, 8)
    o = bvh["order"]
    osc = oracle.Scene(node_min=bvh["node_min"], node_max=bvh["node_max"], left=bvh["left"], right=bvh["right"],
                       start=bvh["start"], count=bvh["count"], v0=v0[o], v1=v1[o], v2=v2[o])
    rt, ridx, ru, rv = oracle.bvh_intersect(osc, ro, rd)
    ridx = np.where(ridx >= 0, o[np.maximum(ridx, 0)], -1)
    sc = _scene(v0, v1, v2, method, leaf)
    t, idx, u, v = sc.trace_closest(ro, rd)
    w = 1.0 - ru - rv
    near_edge = (ridx >= 0) & (np.minimum(np.minimum(ru, rv), w) < 1e-6)
    mism = idx != ridx
    ties = np.zeros(len(ro), bool)
    for i in np.nonzero(mism & ~near_edge)[0]:
        if idx[i] >= 0 and ridx[i] >= 0:
            tt, _, _ = oracle.tri_intersect(ro[i:i + 1], rd[i:i + 1], v0[idx[i]:idx[i] + 1], v1[idx[i]:idx[i] + 1],
                                            v2[idx[i]:idx[i] + 1])
            ties[i] = tt[0] == rt[i]
    excluded = near_edge | ties
    bad = mism & ~excluded
    assert not bad.any(), f"{bad.sum()} id mismatches outside exclusions, e.g. ray {np.nonzero(bad)[0][:5]}"
    ok = (idx >= 0) & ~excluded
    np.testing.assert_allclose(t[ok], rt[ok], rtol=1e-5)
    np.testing.assert_allclose(u[ok], ru[ok], rtol=1e-5, atol=1e-6)
    np.testing.assert_allclose(v[ok], rv[ok], rtol=1e-5, atol=1e-6)
    return dict(rays=len(ro), hits=int((ridx >= 0).sum()), excluded_edge=int(near_edge.sum()),
                excluded_ties=int(ties.sum()), bit_exact_t=bool(np.array_equal(t[ok].view(np.uint32),
                                                                               rt[ok].view(np.uint32))))


def test_lbvh_golden_rays():
    g = np.load(os.path.join(GOLD, "traversal.npz"))
    for case in g["case_names"]:
        c = {k.split("/", 1)[1]: g[k] for k in g.files if k.startswith(f"{case}/")}
        r = _parity(c["v0"], c["v1"], c["v2"], c["ro"], c["rd"])
        assert r["bit_exact_t"]


def test_lbvh_hit_ids_on_seeded_ray_set_displaced_mesh():
    pos, f = gs.icosphere(6)
    rng = np.random.default_rng(11)
    pos = pos * (1 + 0.05 * rng.standard_normal(len(pos)))[:, None]
    v0, v1, v2 = (pos[f[:, k]].astype(np.float32) for k in range(3))
    # rays from a shell toward the mesh plus fully random rays
    n = 60000
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    ro = (d * 3.0).astype(np.float32)
    tgt = rng.uniform(-0.9, 0.9, size=(n, 3))
    rd = tgt - ro
    rd = (rd / np.linalg.norm(rd, axis=1, keepdims=True)).astype(np.float32)
    ro2, rd2 = gs.random_rays(20000, 12, spread=0.8)
    r = _parity(v0, v1, v2, np.concatenate([ro, ro2]), np.concatenate([rd, rd2]))
    assert r["hits"] > 0.8 * n
    assert r["excluded_edge"] + r["excluded_ties"] < 0.001 * r["rays"]
    assert r["bit_exact_t"]


def test_lbvh_soup_and_leaf_sizes():
    v0, v1, v2 = gs.soup_triangles(30000, 31)
    ro, rd = gs.random_rays(30000, 32)
    for leaf in (1, 2, 4, 8):
        _parity(v0, v1, v2, ro, rd, leaf=leaf)


def test_any_hit_matches_oracle():
    v0, v1, v2 = gs.soup_triangles(20000, 41)
    ro, rd = gs.random_rays(40000, 42)
    tmax = np.random.default_rng(43).uniform(0.01, 2.0, len(ro)).astype(np.float32)
    bvh = oracle.bvh_build_morton(v0, v1, v2, 8)
    o = bvh["order"]
    osc = oracle.Scene(node_min=bvh["node_min"], node_max=bvh["node_max"], left=bvh["left"], right=bvh["right"],
                       start=bvh["start"], count=bvh["count"], v0=v0[o], v1=v1[o], v2=v2[o])
    ref = oracle.bvh_occluded(osc, ro, rd, tmax)
    for method in (nat.RX_BVH_REFERENCE, nat.RX_BVH_LBVH_SAH):
        sc = _scene(v0, v1, v2, method, 8 if method == nat.RX_BVH_REFERENCE else 4)
        got = sc.trace_any(ro, rd, tmax)
        # the any-hit decision only differs when a hit sits exactly at tmax
        assert (got != ref).sum() <= 2


def test_empty_and_degenerate_inputs():
    sc = nat.NativeScene()
    sc.set_materials([0], [[0.5, 0.5, 0.5]], [0.0], [1.0], [0.0])
    sc.set_triangles(np.zeros((0, 3)), np.zeros((0, 3)), np.zeros((0, 3)))
    t, idx, _, _ = sc.trace_closest(np.zeros((3, 3)), np.tile([0, 0, 1.0], (3, 1)))
    assert (idx == -1).all() and (t == 1e9).all()
    # zero-length rays and degenerate (zero-area) triangles
    v0 = np.zeros((4, 3), np.float32)
    sc2 = _scene(v0, v0, v0, nat.RX_BVH_LBVH_SAH, 4)
    t, idx, _, _ = sc2.trace_closest(np.ones((2, 3)), np.zeros((2, 3)))
    assert (idx == -1).all()


def _benchmark_scene_rays(world, host, osc, n_cam=100000, n_sec=100000, n_shell=50000, seed=2025):
    """Seeded ray set on the benchmark scene: jittered camera rays through the
    1920x1080 frame of the scene's own camera, secondary rays leaving the
    camera rays' first hits (origin offset 1e-4 along the facing normal, as
    trace.py:234 does; cosine-weighted directions) and shell rays aimed into
    the sphere cloud."""
    import math
    rng = np.random.default_rng(seed)
    cam = world.active_camera
    tan = math.tan(math.radians(cam.fov) / 2)
    fwd, right, up = (np.array([c.x, c.y, c.z], np.float64) for c in (cam.forward, cam.right, cam.up))
    px = rng.uniform(0, 1920, n_cam)
    py = rng.uniform(0, 1080, n_cam)
    su = (2.0 * px / 1920 - 1.0) * cam.aspect_ratio * tan
    sv = (1.0 - 2.0 * py / 1080) * tan
    d = fwd[None] + su[:, None] * right[None] + sv[:, None] * up[None]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    ro_c = np.tile(np.array([cam.position.x, cam.position.y, cam.position.z], np.float32), (n_cam, 1))
    rd_c = d.astype(np.float32)
    first = oracle.scene_intersect(osc, ro_c, rd_c)
    hit = np.nonzero(first["idx"] >= 0)[0]
    pick = rng.choice(hit, n_sec)
    nrm = first["normal"][pick].astype(np.float64)
    flip = (nrm * rd_c[pick]).sum(1) > 0
    nrm[flip] *= -1
    p = ro_c[pick] + rd_c[pick] * first["t"][pick][:, None]
    ro_s = (p + nrm * 1e-4).astype(np.float32)
    rnd = rng.normal(size=(n_sec, 3))
    rnd /= np.linalg.norm(rnd, axis=1, keepdims=True)
    rd_s = nrm + rnd
    rd_s /= np.maximum(np.linalg.norm(rd_s, axis=1, keepdims=True), 1e-12)
    g = rng.normal(size=(n_shell, 3))
    g /= np.linalg.norm(g, axis=1, keepdims=True)
    ro_h = g * 3.5
    tgt = rng.uniform(-0.8, 0.8, (n_shell, 3))
    rd_h = tgt - ro_h
    rd_h /= np.linalg.norm(rd_h, axis=1, keepdims=True)
    ro = np.concatenate([ro_c, ro_s, ro_h.astype(np.float32)])
    rd = np.concatenate([rd_c, rd_s.astype(np.float32), rd_h.astype(np.float32)])
    return np.ascontiguousarray(ro, np.float32), np.ascontiguousarray(rd, np.float32)


def test_benchmark_scene_hit_ids_match_reference_traversal():
    """The benchmark scene itself (327,680 displaced-icosphere triangles,
    64 spheres as LBVH leaves, the light quad): 250,000 seeded rays through
    rx_scene_intersect against the oracle's scene_intersect over the
    reference Morton tree and its linear object scan
    (rendering/taichi/intersect.py:249-309).  Hit ids (triangle or object
    slot) are bit-exact outside counted edge / exact-tie exclusions
    (< 0.1 %), t / u / v agree to 1e-5 relative."""
    import workloads
    from helpers import oracle_scene
    from rendering.taichi.extractor import HostScene, build_device_scene, slot_arrays
    world = workloads.displaced_icosphere_scene()
    host = HostScene(world)
    b = host.batch
    assert b.triangle_count == 327682 and len(host.slots) == 64
    osc = oracle_scene(host, False)
    order = oracle.bvh_build_morton(b.v0, b.v1, b.v2, 8)["order"]
    objs = oracle.Scene(objects=slot_arrays(host.slots))
    ro, rd = _benchmark_scene_rays(world, host, osc)
    assert len(ro) >= 200000
    ref = oracle.scene_intersect(osc, ro, rd)
    ds = build_device_scene(world, method="lbvh")
    got = ds.native.intersect(ro, rd)
    assert (got["kind"] == 2).any(), "spheres are expected as BVH leaves"
    r = parity.compare_closest(got, ref, order, ro, rd, b.v0, b.v1, b.v2, objects_scene=objs)
    print("benchmark-scene parity:", r)
    assert r["hits"] > 0.3 * r["rays"] and r["object_hits"] > 1000
    assert r["excluded_edge"] + r["excluded_ties"] < 0.001 * r["rays"]
    assert r["t_bit_exact"]


@pytest.mark.parametrize("n", [1, 33, 1184, 1185, 4000, 37_887, 37_889])
def test_short_queries_equal_long_ones(n):
    """Fewer rays per warp below 37,888 of them: every ray's answer is the one
    it has in a query of 60,000, whatever the number of lanes a warp uses."""
    v0, v1, v2 = gs.soup_triangles(3000, 11)
    sc = _scene(v0, v1, v2, nat.RX_BVH_LBVH_SAH, 4)
    rng = np.random.default_rng(2)
    ro = rng.normal(size=(60_000, 3)).astype(np.float32) * 2
    rd = rng.normal(size=(60_000, 3)).astype(np.float32)
    rd /= np.linalg.norm(rd, axis=1, keepdims=True)
    tm = rng.uniform(0.1, 4.0, 60_000).astype(np.float32)
    for a, b in zip(sc.trace_closest(ro, rd), sc.trace_closest(ro[-n:], rd[-n:])):
        assert np.array_equal(a[-n:].view(np.int32), b.view(np.int32))
    assert np.array_equal(sc.trace_any(ro, rd, tm)[-n:], sc.trace_any(ro[-n:], rd[-n:], tm[-n:]))


@pytest.mark.parametrize("n,scale,offset", [(1, 1.0, 0.0), (2, 0.01, 0.0), (5, 1.0, 50.0), (33, 100.0, 0.0),
                                            (3000, 1.0, 0.0), (3000, 0.05, 20.0), (3000, 100.0, 50.0)])
def test_wide_nodes_find_what_the_reference_tree_finds(n, scale, offset):
    """The 4-wide traversal of ray queries (both planes of an axis in one
    load) against the binary tree with the reference's slab test: the same t
    bit for bit on every ray (the triangle test is the same; a box may only
    cost a visit), over scene sizes, positions and axis-parallel directions."""
    rng = np.random.default_rng(n + int(scale * 100) + int(offset))
    ctr = rng.uniform(-1, 1, (n, 1, 3))
    tri = ((ctr + rng.normal(0, 0.1, (n, 3, 3))) * scale + offset).astype(np.float32)
    m = 20000
    aim = tri[rng.integers(0, n, m)].mean(axis=1) + rng.normal(0, 0.05 * scale, (m, 3))
    rd = rng.normal(size=(m, 3))
    axis = rng.integers(0, 3, m // 4)
    rd[:m // 4] = 0.0
    rd[np.arange(m // 4), axis] = rng.choice([-1.0, 1.0], m // 4)
    rd = (rd / np.linalg.norm(rd, axis=1, keepdims=True)).astype(np.float32)
    ro = (aim - rd * rng.uniform(0.0, 3.0 * scale, (m, 1))).astype(np.float32)
    wide = _scene(tri[:, 0], tri[:, 1], tri[:, 2], nat.RX_BVH_LBVH_SAH, 4)
    ref = _scene(tri[:, 0], tri[:, 1], tri[:, 2], nat.RX_BVH_REFERENCE, 4)
    t0, t1 = wide.trace_closest(ro, rd)[0], ref.trace_closest(ro, rd)[0]
    assert (t1 < 1e9).sum() > m // 50
    np.testing.assert_array_equal(t0.view(np.uint32), t1.view(np.uint32))
    tmax = rng.uniform(0.0, 3.0 * scale, m).astype(np.float32)
    np.testing.assert_array_equal(wide.trace_any(ro, rd, tmax), ref.trace_any(ro, rd, tmax))


@pytest.mark.parametrize("n", [8_001, 20_000, 36_704, 36_705])
def test_query_lanes_up_to_whole_warps(n):
    """Odd numbers of rays per warp (7, 17, 31, then 32 from 36,705 rays on
    148 SMs), the hits with normals among the queries: the answers of a query
    of 60,000 rays."""
    v0, v1, v2 = gs.soup_triangles(3000, 11)
    sc = _scene(v0, v1, v2, nat.RX_BVH_LBVH_SAH, 4)
    rng = np.random.default_rng(2)
    ro = rng.normal(size=(60_000, 3)).astype(np.float32) * 2
    rd = rng.normal(size=(60_000, 3)).astype(np.float32)
    rd /= np.linalg.norm(rd, axis=1, keepdims=True)
    tm = rng.uniform(0.1, 4.0, 60_000).astype(np.float32)
    for a, b in zip(sc.trace_closest(ro, rd), sc.trace_closest(ro[-n:], rd[-n:])):
        assert np.array_equal(a[-n:].view(np.int32), b.view(np.int32))
    assert np.array_equal(sc.trace_any(ro, rd, tm)[-n:], sc.trace_any(ro[-n:], rd[-n:], tm[-n:]))
    whole, part = sc.intersect(ro, rd), sc.intersect(ro[-n:], rd[-n:])
    for k in whole:
        assert np.array_equal(whole[k][-n:].view(np.int32), part[k].view(np.int32)), k
