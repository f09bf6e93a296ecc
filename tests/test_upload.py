"""Upload of large meshes: the triangles are packed on the device in parts, whose memory is bounded."""
import numpy as np
import pytest

import pathed


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 262143, 262144, 262145, 524289])
def test_triangles_on_both_sides_of_a_part(n):
    """a grid of small triangles: ids and materials as given, and the distances of the tree that the host builds
    from its own arrays"""
    side = int(np.ceil(np.sqrt(n)))
    k = np.arange(n)
    x, y = (k % side).astype(np.float32), (k // side).astype(np.float32)
    v = np.zeros((n, 3, 3), np.float32)
    v[:, 0, 0], v[:, 0, 1] = x + 0.1, y + 0.1
    v[:, 1, 0], v[:, 1, 1] = x + 0.9, y + 0.1
    v[:, 2, 0], v[:, 2, 1] = x + 0.1, y + 0.9
    nrm = np.zeros_like(v)
    nrm[:, :, 2] = 1
    pick = np.unique(np.clip(np.concatenate([np.arange(-3, 4) + e for e in (0, 262144, 524288, n - 1, n // 2)]), 0, n - 1))
    o = np.stack([x[pick] + 0.2, y[pick] + 0.2, np.full(len(pick), 2)], 1).astype(np.float32)
    d = np.tile(np.float32([0, 0, -1]), (len(pick), 1))
    hits = []
    for builder in (0, 2):  # 2: the tree too is built from the packed vertices
        s = pathed.Session(8, 8)
        s.set_bvh_builder(builder)
        s.load_arrays(tri_vertices=v, tri_normals=nrm, tri_materials=(k % 3).astype(np.int32), material_types=[0] * 3,
                      material_albedo=[[0.5] * 3] * 3, material_emit=[[0] * 3] * 3, material_ior=[1.0] * 3,
                      material_alpha=[0.1] * 3)
        hits.append(s.trace_rays(o, d, 0.0, 1e6, with_bary=True))
        s.close()
    for g in hits:
        assert np.array_equal(g["prim_id"], pick)
        assert np.array_equal(g["mat_id"], pick % 3)
    for key in ("t", "bary"):
        assert np.array_equal(hits[0][key], hits[1][key])


@pytest.mark.gpu
def test_scratch_memory_of_a_large_mesh():
    """What a session of the 1.31M-triangle mesh keeps on the device: records, leaf entries, nodes, environment
    and stacks (about 340 MB), without the 100 MB that one-piece packing of its triangles left behind."""
    import torch

    torch.cuda.synchronize()
    s = pathed.Session(8, 8)
    s.load_config(2)
    s.hit_test(0, 0)
    before = torch.cuda.mem_get_info()[0]
    s.close()
    kept = torch.cuda.mem_get_info()[0] - before
    assert kept < 400e6, kept
