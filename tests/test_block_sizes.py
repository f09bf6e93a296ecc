"""Traversal blocks of every size that set_launch takes: the image of the default blocks, or an error
that leaves the session usable where an SM has not the registers."""
import numpy as np
import pytest

import pathed


def _image(s):
    s.reset()
    s.render(2)
    return s.readback().copy()


@pytest.mark.gpu
@pytest.mark.parametrize("width,option,largest", [(2, "", 1024), (4, "", 1024), (4, "quantized", 1024), (4, "watertight", 1024),
                                                  (8, "", 768), (8, "quantized", 896), (8, "watertight", 768)])
def test_largest_blocks(width, option, largest):
    s = pathed.Session(61, 47)
    s.set_bvh(width, 4)
    s.set_bvh_quantized(option == "quantized")
    s.set_watertight(option == "watertight")
    s.load_config(3, level=4)
    s.set_max_depth(4)
    ref = _image(s)
    for extend, shadow in ((largest, largest), (largest, 32), (32, largest)):
        s.set_launch(block_extend=extend, block_shadow=shadow)
        assert np.array_equal(_image(s), ref), (extend, shadow)
    for block in range(largest + 32, 1025, 32):
        s.set_launch(block_extend=block, block_shadow=128)
        with pytest.raises(pathed.PathedError):
            s.render(2)
    s.set_launch(block_extend=128, block_shadow=128)
    assert np.array_equal(_image(s), ref)
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("graph", [1, 2])
def test_sessions_of_different_blocks(graph):
    """The kernels' shared-memory limit is the process's: a session of smaller blocks does not lower it under
    another's frames."""
    def session(block):
        s = pathed.Session(61, 47)
        s.load_config(0)
        s.set_launch(block_extend=block, block_shadow=block, use_graph=graph)
        return s

    small = session(128)
    ref = {spp: None for spp in (1, 2, 3)}
    for spp in ref:
        small.reset()
        small.render(spp)
        ref[spp] = small.readback().copy()
    a, b = session(1024), session(512)
    for spp in ref:  # another spp each time: the frame is launched, or captured, anew
        for s in (a, b, a):
            s.reset()
            s.render(spp)
            assert np.array_equal(s.readback(), ref[spp]), spp
    for s in (small, a, b):
        s.close()
