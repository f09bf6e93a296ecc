"""Traversal stacks that run past their shared-memory part, on every route that has its own part of the
global memory behind them: several workers of one host call, the allocation-free call, the shadow stage.
And frames whose last queries are shared among a warp's lanes against frames where they are not."""
import numpy as np
import pytest

import pathed
from _util import FLT_MAX

SHARED = 12  # entries of a lane in shared memory


def _sheets(n):
    """n large triangles one behind the other: a ray along z leaves width - 1 entries behind per level."""
    z = np.arange(n, dtype=np.float32) * np.float32(0.01)
    v = np.zeros((n, 3, 3), np.float32)
    v[:, 0, :2], v[:, 1, :2], v[:, 2, :2] = (-30, -20), (30, -20), (0, 40)
    v[:, :, 2] = z[:, None]
    nrm = np.zeros_like(v)
    nrm[:, :, 2] = -1
    return v, nrm


def _load(s, v, nrm, **more):
    s.load_arrays(tri_vertices=v, tri_normals=nrm, tri_materials=np.zeros(len(v), np.int32), material_types=[0],
                  material_albedo=[[0.5, 0.5, 0.5]], material_emit=[[0, 0, 0]], material_ior=[1.0], material_alpha=[0.1], **more)


def _static(s, o, d, tmin, tmax):
    n = len(o)
    out = [np.zeros(n, np.int32) for _ in range(3)] + [np.zeros(n, np.float32)]
    s._check(pathed.lib.pt_trace_rays_static(s._h, o.ctypes.data, d.ctypes.data, tmin.ctypes.data, tmax.ctypes.data, n,
                                             *[a.ctypes.data for a in out], None))
    return dict(zip(("prim_type", "prim_id", "mat_id", "t"), out))


@pytest.mark.gpu
@pytest.mark.parametrize("width,n", [(2, 60000), (4, 12000), (8, 12000)])
def test_spilled_stacks_on_every_route(oracle_lib, width, n):
    v, nrm = _sheets(n)
    s = pathed.Session(32, 32)
    s.set_bvh(width, 1)
    _load(s, v, nrm)
    # a ray through all sheets leaves this many entries on its way down to the nearest
    assert (width - 1) * (s.counts().bvh_depth - 1) > SHARED
    rng = np.random.default_rng(width)
    m = 150001  # eight workers
    o = np.zeros((m, 3), np.float32)
    o[:, :2] = rng.uniform(-5, 5, (m, 2))
    o[:, 2] = -1
    d = np.tile(np.float32([0, 0, 1]), (m, 1))
    tmin = np.where(rng.random(m) < 0.5, 0, rng.uniform(0, n * 0.01, m)).astype(np.float32)
    tmax = np.full(m, FLT_MAX, np.float32)
    big = s.trace_rays(o, d, tmin, tmax)
    occ = s.occluded(o, d, tmin, tmax)
    k = 300
    ref = oracle_lib.trace(oracle_lib.scene(s.export_scene()), o[:k], d[:k], tmin[:k], tmax[:k])
    for key in ("prim_type", "prim_id", "mat_id", "t"):
        assert np.array_equal(big[key][:k], ref[key]), key
    assert np.array_equal(occ, (big["prim_type"] >= 0).astype(np.int32))
    for a in range(0, m, 65536):  # one worker, then the allocation-free route
        part = [x[a:a + 65536].copy() for x in (o, d, tmin, tmax)]
        for got in (s.trace_rays(*part), _static(s, *part)):
            for key in ("prim_type", "prim_id", "mat_id", "t"):
                assert np.array_equal(got[key], big[key][a:a + 65536]), key
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("width,n", [(2, 12000), (4, 3000), (8, 3000)])
@pytest.mark.parametrize("order", [1, 2])
def test_spilled_stacks_in_the_shadow_stage(oracle_lib, width, n, order):
    """A floor lit through a stack of upright sheets that stop short of the light's rays: each shadow ray enters
    their boxes and finds nothing, or is occluded; the image is the oracle's."""
    v = np.zeros((n, 3, 3), np.float32)
    x = np.linspace(-1, 1, n, dtype=np.float32)
    rng = np.random.default_rng(n)
    # slivers across the light's way, of random heights: boxes overlap along every shadow ray
    v[:, 0] = np.stack([x, np.full(n, 1.0), np.full(n, -2.0)], 1)
    v[:, 1] = np.stack([x, rng.uniform(1.0, 1.4, n), np.full(n, 2.0)], 1)
    v[:, 2] = np.stack([x + 0.001, np.full(n, 1.01), np.full(n, 2.0)], 1)
    floor = np.float32([[[-3, 0, -3], [3, 0, -3], [3, 0, 3]], [[-3, 0, -3], [3, 0, 3], [-3, 0, 3]]])
    lamp = np.float32([[[2.6, 1.2, -0.3], [2.6, 1.5, 0.3], [2.6, 1.2, 0.3]]])
    tri = np.concatenate([v, floor, lamp])
    nrm = np.zeros_like(tri)
    nrm[:n, :, 0], nrm[n:n + 2, :, 1], nrm[n + 2:, :, 0] = -1, 1, -1
    mats = np.concatenate([np.zeros(n + 2), [1]]).astype(np.int32)
    s = pathed.Session(40, 30)
    s.set_bvh(width, 1)
    s.load_arrays(tri_vertices=tri, tri_normals=nrm, tri_materials=mats, material_types=[0, 0],
                  material_albedo=[[0.7, 0.6, 0.5], [0, 0, 0]], material_emit=[[0, 0, 0], [9, 9, 9]], material_ior=[1.0] * 2,
                  material_alpha=[0.1] * 2)
    s.set_camera((-2.8, 0.9, 0.2), (0, 0.6, 0), (0, 1, 0), 0.9)
    s.set_max_depth(2)
    s.set_nee(True)
    s.set_launch(shadow_order=order)
    assert (width - 1) * (s.counts().bvh_depth - 1) > SHARED or width == 2
    s.render(2)
    img = s.readback().reshape(-1, 3).astype(np.float64)
    sc = s.export_scene()
    mean, _, _ = oracle_lib.render(oracle_lib.scene(sc), sc["camera"], 40, 30, np.arange(1200, dtype=np.int32), 2, 2, nee=True,
                                   seed=0x5EED, sample_base=0, trace_once=True)
    rel = np.abs(img - mean) / (np.abs(mean) + 1e-3)
    assert np.mean(np.all(rel < 1e-3, axis=1)) >= 0.99
    s.close()


def _frames(s, spp=2):
    """Renders the same frame with its last queries shared and, counting each query's work, not."""
    for counters in (False, True):
        s.set_profiling(False, counters)
        s.reset()
        s.render(spp)
        yield counters


@pytest.mark.gpu
@pytest.mark.parametrize("width,option", [(2, ""), (4, ""), (4, "quantized"), (4, "watertight"), (8, ""), (8, "quantized")])
@pytest.mark.parametrize("config", [2, 3])
def test_frames_with_and_without_sharing(config, width, option):
    s = pathed.Session(97, 61)
    s.set_bvh(width, 2)
    s.set_bvh_quantized(option == "quantized")
    s.set_watertight(option == "watertight")
    s.load_config(config, level=7)
    s.set_max_depth(6)
    assert s.counts().bvh_depth >= 6
    for nee in (True, False):
        s.set_nee(nee)
        a, b = [s.readback().copy() for _ in _frames(s)]
        assert np.array_equal(a, b), nee
    s.close()


@pytest.mark.gpu
def test_guided_frames_with_and_without_sharing():
    s = pathed.Session(97, 61)
    s.load_config(3, level=6)
    s.set_max_depth(6)
    s.set_guide_options(steps_per_frame=4, lr=1e-4, warmup_steps=0)
    s.set_guiding(True)
    s.render(1)
    assert s.counts().bvh_depth >= 6
    params = s.guide_params()
    images = []
    for counters in (False, True):
        s.set_profiling(False, counters)
        s.set_guide_params(params)
        s.reset()
        s.render(1)
        images.append(s.readback().copy())
    assert np.array_equal(*images)
    s.close()


@pytest.mark.gpu
def test_batched_frames_with_and_without_sharing():
    specs = pathed.batch_generate(5, 4)
    for k, b in enumerate(specs):
        b.update(level=min(b["level"], 6), width=64, height=64, spp=2, guided=0)
    s = pathed.Session(64, 64)
    s.load_batch(specs)
    images = [[s.batch_readback(k).copy() for k in range(4)] for _ in _frames(s, 1)]
    for a, b in zip(*images):
        assert np.array_equal(a, b)
    s.close()
