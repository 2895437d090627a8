"""Colours an edit takes and refuses."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_set_voxel_colour_types(yoxel_mod):
    """Colours as plain integers, numpy integers and floats give the same
    attribute; one out of range is refused."""
    dyn = yoxel_mod.DynamicSVO(4096, 4096)
    for i, rgb in enumerate([(7, 200, 31), np.array([7, 200, 31]), (7.9, 200.0, 31.2)]):
        dyn.set_voxel(5, 3 * i, 4, 5, rgb=rgb, normal=(-3, 100, 0))
    attrs = dyn.host_arrays()[2]
    assert len(attrs) == 3 and attrs[0].tobytes() == attrs[1].tobytes() == attrs[2].tobytes()
    assert attrs[0].tobytes() == bytes([7, 200, 31, 255, 253, 100, 0, 0])
    with pytest.raises((OverflowError, ValueError)):
        dyn.set_voxel(5, 1, 1, 1, rgb=(300, 0, 0))
