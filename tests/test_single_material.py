"""The shade kernel of scenes whose surfaces all have one material type gives the images of the
per-class kernels (material sorting on) bit for bit, for every type, and follows material edits."""
import numpy as np
import pytest

import pathed


def _image(s, spp=5, **launch):
    s.set_launch(**launch)
    s.reset()
    s.render(spp)
    return s.readback().copy()


@pytest.mark.gpu
@pytest.mark.parametrize("mtype", [pathed.LAMBERTIAN, pathed.MIRROR, pathed.GLASS, pathed.MICROFACET, pathed.METAL])
@pytest.mark.parametrize("size", [(1, 1), (67, 45)])
def test_one_material_equals_class_kernels(mtype, size):
    s = pathed.Session(*size)
    s.load_config(2, level=3)  # one material under an environment map
    s.set_material(0, mtype)
    if mtype == pathed.LAMBERTIAN:
        s.set_material(0, mtype, albedo=(0.6, 0.5, 0.4))
    sorted_ = _image(s, sort_materials=1, split_shade=1)
    for split in (1, 2, 3):
        assert np.array_equal(_image(s, sort_materials=2, split_shade=split), sorted_), split
    assert np.array_equal(_image(s, sort_materials=1, split_shade=2), sorted_)
    assert np.all(np.isfinite(sorted_))
    s.close()


@pytest.mark.gpu
def test_a_second_material_leaves_the_single_material_kernel():
    s = pathed.Session(64, 48)
    s.load_config(0)  # all Lambertian
    one = _image(s, sort_materials=2, split_shade=1)
    s.set_material(0, pathed.MIRROR)
    mixed = _image(s, sort_materials=2, split_shade=1)
    assert np.array_equal(mixed, _image(s, sort_materials=1, split_shade=1))
    s.set_material(0, pathed.LAMBERTIAN)
    s.set_material(0, pathed.LAMBERTIAN, albedo=(0.73, 0.73, 0.73))
    assert np.array_equal(_image(s, sort_materials=2, split_shade=1), one)
    s.close()
