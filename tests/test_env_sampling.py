"""Environment importance sampling through the CDFs' cut points: the same texel as a search of the
whole CDF (the oracle's linear scan, as the reference's), for map sizes around and far from the 256 cuts
of a row, with empty rows and texels that hold most of the mass."""
import numpy as np
import pytest

import pathed


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(1, 1), (2, 3), (1, 257), (255, 2), (5, 1000), (300, 256), (64, 2048)])
def test_images_match_the_oracle(oracle_lib, h, w):
    rng = np.random.default_rng(h * 4096 + w)
    env = np.ones((h, w, 4), np.float32)
    env[..., :3] = np.exp(rng.normal(0, 1, (h, w, 1)))
    if h > 2:
        env[rng.integers(0, h, max(1, h // 4)), :, :3] = 0  # empty rows
    if w > 2:
        env[:, rng.integers(0, w, max(1, w // 3)), :3] = 0
        env[h // 2, w // 2, :3] = 50.0 * np.sqrt(h * w)
    src = pathed.Session(8, 8)
    src.load_config(2, level=2)
    a = src.export_scene()
    src.close()
    s = pathed.Session(48, 36)
    s.load_arrays(tri_vertices=a["tri_vertices"], tri_normals=a["tri_normals"], tri_materials=a["tri_materials"],
                  material_types=[pathed.LAMBERTIAN], material_albedo=[[0.8, 0.7, 0.6]], material_emit=[[0, 0, 0]],
                  material_ior=[1.0], material_alpha=[0.1], env_rgba=env)
    c = a["camera"]
    s.set_camera(c[:3], c[3:6], c[6:9], float(c[9]))
    s.set_max_depth(3)
    s.set_nee(True)
    s.render(4)
    img = s.readback().reshape(-1, 3).astype(np.float64)
    sc = s.export_scene()
    mean, _, _ = oracle_lib.render(oracle_lib.scene(sc), sc["camera"], 48, 36, np.arange(48 * 36, dtype=np.int32), 4, 3,
                                   nee=True, seed=0x5EED, sample_base=0, trace_once=True)
    rel = np.abs(img - mean) / (np.abs(mean) + 1e-3)
    assert np.mean(np.all(rel < 1e-3, axis=1)) >= 0.99
    s.close()
