"""Colours and normals that an edit takes: packed as the numpy assignment into the
attribute record gives them, or refused as it refuses them (no GPU: the library
call is replaced)."""
import ctypes as C

import numpy as np
import pytest


def edit(yoxel_mod, monkeypatch, rgb, normal):
    """The attribute that set_voxel hands to the library."""
    from yoxel import dynamic
    got = []

    class Lib:
        @staticmethod
        def yv_svo_dynamic_set_voxel(h, depth, x, y, z, a):
            got.append(a if isinstance(a, bytes) else C.string_at(a, 8))
            return dynamic.L.YV_OK

    monkeypatch.setattr(dynamic.L, "lib", Lib)
    dyn = object.__new__(yoxel_mod.DynamicSVO)
    dyn._h = None
    dyn.set_voxel(5, 1, 2, 3, rgb=rgb, normal=normal)
    return got[0]


def by_numpy(rgb, normal):
    from yoxel import ATTR_DTYPE
    at = np.zeros(1, ATTR_DTYPE)
    at["rgb"][0] = [rgb[0], rgb[1], rgb[2], 255]
    at["n"][0] = [normal[0], normal[1], normal[2], 0]
    return at.tobytes()


def colours():
    import torch

    class Index:  # an integer by its conversions
        def __init__(self, v):
            self.v = v

        def __index__(self):
            return self.v

        def __int__(self):
            return self.v

        def __float__(self):
            return float(self.v)

    return {
        "ints": (7, 200, 31),
        "numpy ints": np.array([7, 200, 31]),
        "numpy bytes": np.array([7, 200, 31], np.uint8),
        "floats": (7.9, 200.0, 31.2),
        "numpy floats": np.array([7.9, 200.0, 31.2], np.float32),
        "float tensor": torch.tensor([7.9, 200.0, 31.0]),
        "int tensor": torch.tensor([7, 200, 31]),
        "0-d float arrays": [np.array(7.9), np.array(200.0), np.array(31.0)],
        "1-element tensors": [torch.tensor([7.0]), torch.tensor([200.0]), torch.tensor([31.0])],
        "bools": (True, False, True),
        "numpy bools": np.array([True, False, True]),
        "index objects": (Index(7), Index(200), Index(31)),
        "bytes": b"\x07\xc8\x1f",
        "out of range": (300, 0, 0),
        "negative": (-1, 0, 0),
        "numpy out of range": np.array([300, -1, 0]),
        "huge": (1 << 80, 0, 0),
        "nan": (float("nan"), 1.0, 2.0),
        "none": (None, 1, 2),
        "text": "123",
        "words": ("a", "b", "c"),
        "rows": np.zeros((3, 2)),
        "too few": (1, 2),
        "not a sequence": 5,
    }


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("name", list(colours()))
def test_as_numpy_takes_or_refuses(yoxel_mod, monkeypatch, name):
    value = colours()[name]
    for rgb, normal in ((value, (-3, 100, 0)), ((7, 200, 31), value)):
        try:
            want = by_numpy(rgb, normal)
        except Exception as e:
            with pytest.raises(type(e)):
                edit(yoxel_mod, monkeypatch, rgb, normal)
        else:
            assert edit(yoxel_mod, monkeypatch, rgb, normal) == want
