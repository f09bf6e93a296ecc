"""The traversal stack's two parts (shared memory, then global memory) and the ray queries' work
distribution, at the sizes where they could go wrong. The expected hits are the oracle's linear scan,
bit for bit: the closest hit is the minimum of a total order, whatever order nodes are visited in."""
import numpy as np
import pytest

import pathed
from _util import FLT_MAX, seeded_rays


def _parallel_sheets(n):
    """n large triangles one behind the other: a ray along z enters every node's every child, so
    the closest-hit stack grows by width - 1 entries per level, past its shared-memory part."""
    z = np.arange(n, dtype=np.float32) * np.float32(0.01)
    v = np.zeros((n, 3, 3), np.float32)
    v[:, 0, :2], v[:, 1, :2], v[:, 2, :2] = (-30, -20), (30, -20), (0, 40)
    v[:, :, 2] = z[:, None]
    nrm = np.zeros_like(v)
    nrm[:, :, 2] = -1
    return v, nrm


@pytest.mark.gpu
@pytest.mark.parametrize("width,leaf", [(2, 1), (4, 1), (4, 4), (8, 1)])
def test_deep_stacks_give_the_scan_s_hits(oracle_lib, width, leaf):
    n = 3000
    v, nrm = _parallel_sheets(n)
    s = pathed.Session(32, 32)
    s.set_bvh(width, leaf)
    s.load_arrays(tri_vertices=v, tri_normals=nrm, tri_materials=np.zeros(n, np.int32), material_types=[0],
                  material_albedo=[[0.5, 0.5, 0.5]], material_emit=[[0, 0, 0]], material_ior=[1.0], material_alpha=[0.1])
    sc = s.export_scene()
    rng = np.random.default_rng(width * 10 + leaf)
    m = 2000
    o = np.zeros((m, 3), np.float32)
    o[:, :2] = rng.uniform(-5, 5, (m, 2))
    o[:, 2] = rng.choice([-1.0, 31.0, 14.9951], m)
    d = rng.normal(0, 0.02, (m, 3)).astype(np.float32)
    d[:, 2] = np.where(o[:, 2] < 0, 1.0, np.where(o[:, 2] > 30, -1.0, rng.choice([-1.0, 1.0], m)))
    tmin = rng.uniform(0, 20, m).astype(np.float32)  # far hits: most of the tree is entered and left behind
    tmax = np.where(rng.random(m) < 0.5, FLT_MAX, tmin + rng.uniform(0, 0.02, m)).astype(np.float32)
    r = oracle_lib.trace(oracle_lib.scene(sc), o, d, tmin, tmax)
    g = s.trace_rays(o, d, tmin, tmax)
    assert (r["prim_type"] >= 0).sum() > m // 4
    for k in ("prim_type", "prim_id", "mat_id", "t"):
        assert np.array_equal(g[k], r[k]), k
    assert np.array_equal(s.occluded(o, d, tmin, tmax), (r["prim_type"] >= 0).astype(np.int32))
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 400003])  # the last is more than stays resident
def test_query_counts(n):
    s = pathed.Session(32, 32)
    s.load_config(3, level=3)
    o, d, tmin, tmax = seeded_rays(s.export_scene(), n + 2, seed=n)
    o, d, tmin, tmax = o[:n], d[:n], tmin[:n], tmax[:n]
    g = s.trace_rays(o, d, tmin, tmax, with_bary=True)
    occ = s.occluded(o, d, tmin, tmax)
    step = 20000  # calls whose rays all start in their warp's first 32
    parts = [s.trace_rays(o[a:a + step], d[a:a + step], tmin[a:a + step], tmax[a:a + step], with_bary=True)
             for a in range(0, n, step)]
    for k in g:
        assert np.array_equal(g[k], np.concatenate([p[k] for p in parts])), k
    assert np.array_equal(occ, (g["prim_type"] >= 0).astype(np.int32))
    s.close()


@pytest.mark.gpu
def test_query_arrays_may_overlap():
    """results written over rays (a call of several chunks): every ray is read first"""
    n = 70001
    s = pathed.Session(32, 32)
    s.load_config(0)
    o, d, tmin, tmax = seeded_rays(s.export_scene(), n, seed=9)
    ref = s.trace_rays(o, d, tmin, tmax)
    out = [np.empty(n, np.int32) for _ in range(3)]
    t = o.reshape(-1)[n:]  # the distances go over the origins' later two thirds
    s._check(pathed.lib.pt_trace_rays(s._h, o.ctypes.data, d.ctypes.data, tmin.ctypes.data, tmax.ctypes.data, n,
                                      out[0].ctypes.data, out[1].ctypes.data, out[2].ctypes.data, t.ctypes.data, None))
    for k, got in zip(("prim_type", "prim_id", "mat_id"), out):
        assert np.array_equal(got, ref[k]), k
    assert np.array_equal(t[:n], ref["t"])
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("width", [2, 4])
def test_ties_when_queries_are_shared(oracle_lib, width):
    """few long queries (fewer than a warp's worth: its idle lanes share them) among coincident
    primitives: the scan's tie rules decide, across the lanes' parts of a query too"""
    n = 1500
    v, nrm = _parallel_sheets(n)
    v, nrm = np.concatenate([v, v[::-1]]), np.concatenate([nrm, nrm[::-1]])  # every sheet twice
    zs = np.repeat(np.arange(0, 15, 0.05, dtype=np.float32), 2)  # and spheres, twice, tangent to sheets
    sph = np.stack([np.zeros_like(zs), np.zeros_like(zs), zs + np.float32(0.5), np.full_like(zs, 0.5)], 1)
    s = pathed.Session(32, 32)
    s.set_bvh(width, 1)
    s.load_arrays(tri_vertices=v, tri_normals=nrm, tri_materials=np.zeros(2 * n, np.int32), spheres=sph,
                  sphere_materials=np.zeros(len(sph), np.int32), material_types=[0], material_albedo=[[0.5, 0.5, 0.5]],
                  material_emit=[[0, 0, 0]], material_ior=[1.0], material_alpha=[0.1])
    assert s.counts().bvh_depth >= 6
    osc = oracle_lib.scene(s.export_scene())
    rng = np.random.default_rng(width)
    for m in (1, 3, 17, 300):
        o = np.zeros((m, 3), np.float32)
        o[:, 2] = -1
        d = np.tile(np.float32([0, 0, 1]), (m, 1))
        tmin = (1 + 0.01 * rng.integers(0, n - 20, m)).astype(np.float32) - np.float32(0.003)
        tmax = np.full(m, FLT_MAX, np.float32)
        r, g = oracle_lib.trace(osc, o, d, tmin, tmax), s.trace_rays(o, d, tmin, tmax)
        for k in ("prim_type", "prim_id", "t"):
            assert np.array_equal(g[k], r[k]), (m, k)
        t1 = tmin + rng.choice([0.002, 0.5], m).astype(np.float32)  # short ones find nothing
        occ = s.occluded(o, d, tmin, t1)
        assert np.array_equal(occ, (oracle_lib.trace(osc, o, d, tmin, t1)["prim_type"] >= 0).astype(np.int32)), m
    s.close()
