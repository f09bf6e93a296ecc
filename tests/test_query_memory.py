"""Ray queries on host arrays of every kind of memory and layout, at the sizes where the route of a
call changes: the same hits as calls of separate pageable arrays."""
import time

import numpy as np
import pytest

import pathed
from _util import seeded_rays


def _session(config=0):
    s = pathed.Session(32, 32)
    s.load_config(config)
    return s


def _trace(s, o, d, tmin, tmax, hits, n):
    """pt_trace_rays on the caller's own arrays (prim_type, prim_id, mat_id, t, bary)."""
    s._check(pathed.lib.pt_trace_rays(s._h, o.ctypes.data, d.ctypes.data, tmin.ctypes.data, tmax.ctypes.data, n,
                                      *[a.ctypes.data for a in hits]))


def _hits(n):
    return [np.zeros(n, np.int32) for _ in range(3)] + [np.zeros(n, np.float32), np.zeros(2 * n, np.float32)]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [16384, 16385, 65536, 65537, 1000003])
def test_results_over_rays(n):
    """results written over the rays they come from, in arrays that overlap in two ways"""
    s = _session()
    o, d, tmin, tmax = seeded_rays(s.export_scene(), n, seed=n)
    ref = _hits(n)
    _trace(s, o, d, tmin, tmax, ref, n)
    o1, d1, tmin1, tmax1 = o.copy(), d.copy(), tmin.copy(), tmax.copy()
    got = _hits(n)
    got[0] = tmin1.view(np.int32)               # types over the near limits
    got[3] = tmax1                              # distances over the far limits
    got[4] = o1.reshape(-1)[n // 2:]            # barycentrics within the origins
    _trace(s, o1, d1, tmin1, tmax1, got, n)
    for k in range(4):
        assert np.array_equal(got[k], ref[k]), k
    assert np.array_equal(got[4][:2 * n], ref[4])
    occ = d.copy()
    s._check(pathed.lib.pt_occluded(s._h, o.ctypes.data, occ.ctypes.data, tmin.ctypes.data, tmax.ctypes.data, n,
                                    occ.ctypes.data))
    assert np.array_equal(occ.reshape(-1)[:n].view(np.int32), (ref[0] >= 0).astype(np.int32))
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 16384, 16385, 200003])
@pytest.mark.parametrize("pageable", [None, 0, 8])  # which of the nine arrays is not page-locked
def test_page_locked_arrays(n, pageable):
    import torch

    s = _session()
    rays = seeded_rays(s.export_scene(), n + 2, seed=n)
    rays = [a[:n].copy() for a in rays]
    ref = _hits(n)
    _trace(s, *rays, ref, n)
    own = [torch.from_numpy(a) if i == pageable else torch.from_numpy(a).pin_memory()
           for i, a in enumerate(rays + _hits(n))]
    got = [a.numpy() for a in own]
    _trace(s, *got[:4], got[4:], n)
    for a, b in zip(got[4:], ref):
        assert np.array_equal(a, b)
    got[4][:] = 7
    s._check(pathed.lib.pt_occluded(s._h, *[a.ctypes.data for a in got[:4]], n, got[4].ctypes.data))
    assert np.array_equal(got[4], (ref[0] >= 0).astype(np.int32))
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 3000, 70001])
def test_device_memory_is_refused(n):
    """an error, as before queries were staged, not a crash of the host's copy"""
    import torch

    s = _session()
    arrays = [*seeded_rays(s.export_scene(), n + 2, seed=5), *_hits(n)]
    arrays = [a[:2 * n].copy() for a in arrays]
    for k in range(9):
        ptr = [a.ctypes.data for a in arrays]
        on_gpu = torch.from_numpy(arrays[k]).cuda()
        ptr[k] = on_gpu.data_ptr()
        with pytest.raises(pathed.PathedError):
            s._check(pathed.lib.pt_trace_rays(s._h, *ptr[:4], n, *ptr[4:]))
        if k < 5:
            with pytest.raises(pathed.PathedError):
                s._check(pathed.lib.pt_occluded(s._h, *ptr[:4], n, ptr[4]))
    _trace(s, *arrays[:4], arrays[4:], n)  # the session goes on
    s.close()


def _copies(s, arrays, n):
    """The copies to and from the GPU that one call makes."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    _trace(s, *arrays[:4], arrays[4:], n)
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        _trace(s, *arrays[:4], arrays[4:], n)
        torch.cuda.synchronize()
    return tuple(sum(e.count for e in p.key_averages() if "Memcpy" in e.key and way in e.key) for way in ("HtoD", "DtoH"))


@pytest.mark.gpu
def test_page_locked_arrays_are_copied_straight():
    """A large call on page-locked arrays leaves the copies to the GPU: one per array, not one per staged chunk."""
    import torch

    n = 200003
    s = _session()
    own = [torch.from_numpy(a.copy()).pin_memory() for a in [*seeded_rays(s.export_scene(), n, seed=3), *_hits(n)]]
    assert _copies(s, [a.numpy() for a in own], n) == (4, 6)  # and the overflow flag
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2049, 16385, 33000, 65536])
def test_medium_calls_are_staged_in_one_piece(n):
    s = _session()
    assert _copies(s, [*seeded_rays(s.export_scene(), n, seed=4), *_hits(n)], n) == (1, 1)
    s.close()


@pytest.mark.gpu
def test_overlapping_arrays_cost_no_page_locking():
    """A large call whose results go over its rays takes as long as its copies and kernel do (about twice
    the separate arrays' time on a B200), not the 26 times that page-locking a staging of its size took."""
    n = 1000000
    s = _session()
    o, d, tmin, tmax = seeded_rays(s.export_scene(), n, seed=1)
    apart, over = _hits(n), _hits(n)
    over[3] = tmax.copy()

    def best(hits, far):
        t = []
        for _ in range(5):
            far[:] = tmax
            t0 = time.perf_counter()
            _trace(s, o, d, tmin, far, hits, n)
            t.append(time.perf_counter() - t0)
        return min(t[1:])

    assert best(over, over[3]) < 8 * best(apart, tmax.copy())
    s.close()
