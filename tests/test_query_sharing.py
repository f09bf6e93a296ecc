"""Ray queries on both sides of the size from which a call shares its last queries among a warp's idle
lanes, on trees deep enough for it at every width, against the oracle's linear scan."""
import numpy as np
import pytest

import pathed
from _util import FLT_MAX


def _sheets(n):
    """n large triangles one behind the other, each twice, and spheres tangent to some: ties everywhere."""
    z = np.arange(n, dtype=np.float32) * np.float32(0.01)
    v = np.zeros((n, 3, 3), np.float32)
    v[:, 0, :2], v[:, 1, :2], v[:, 2, :2] = (-30, -20), (30, -20), (0, 40)
    v[:, :, 2] = z[:, None]
    nrm = np.zeros_like(v)
    nrm[:, :, 2] = -1
    zs = np.repeat(np.arange(0, n * 0.01, 0.05, dtype=np.float32), 2)
    sph = np.stack([np.zeros_like(zs), np.zeros_like(zs), zs + np.float32(0.5), np.full_like(zs, 0.5)], 1)
    return np.concatenate([v, v[::-1]]), np.concatenate([nrm, nrm[::-1]]), sph


@pytest.mark.gpu
@pytest.mark.parametrize("width,n,quantized", [(2, 1500, False), (4, 3000, False), (4, 3000, True), (8, 20000, False),
                                               (8, 20000, True)])
def test_ties_on_both_sides_of_sharing(oracle_lib, width, n, quantized):
    v, nrm, sph = _sheets(n)
    s = pathed.Session(32, 32)
    s.set_bvh(width, 1)
    s.set_bvh_quantized(quantized)
    s.load_arrays(tri_vertices=v, tri_normals=nrm, tri_materials=np.zeros(2 * n, np.int32), spheres=sph,
                  sphere_materials=np.zeros(len(sph), np.int32), material_types=[0], material_albedo=[[0.5, 0.5, 0.5]],
                  material_emit=[[0, 0, 0]], material_ior=[1.0], material_alpha=[0.1])
    assert s.counts().bvh_depth >= 6
    osc = oracle_lib.scene(s.export_scene())
    rng = np.random.default_rng(width)
    most = 1100
    o = np.zeros((most, 3), np.float32)
    o[:, 2] = -1
    d = np.tile(np.float32([0, 0, 1]), (most, 1))
    d[most // 2:, :2] = rng.normal(0, 0.02, (most - most // 2, 2))
    tmin = (1 + 0.01 * rng.integers(0, n - 20, most)).astype(np.float32) - np.float32(0.003)
    tmax = np.full(most, FLT_MAX, np.float32)
    t1 = tmin + rng.choice([0.002, 0.5], most).astype(np.float32)  # short ones find nothing
    r = oracle_lib.trace(osc, o, d, tmin, tmax)
    occluded = (oracle_lib.trace(osc, o, d, tmin, t1)["prim_type"] >= 0).astype(np.int32)
    for m in (1, 9, 1023, 1024, most):
        g = s.trace_rays(o[:m], d[:m], tmin[:m], tmax[:m])
        for k in ("prim_type", "prim_id", "mat_id", "t"):
            assert np.array_equal(g[k], r[k][:m]), (m, k)
        assert np.array_equal(s.occluded(o[:m], d[:m], tmin[:m], t1[:m]), occluded[:m]), m
    s.close()
