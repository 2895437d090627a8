"""GPU brick-pool build against the host builder where its passes have edges:
single points on rows', cells' and words' borders, arrays that are not aligned
for the wide loads, the apron neighbour tables of device pools."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def equal_volumes(a, b):
    assert a.nbricks == b.nbricks and a.ngrids == b.ngrids
    np.testing.assert_array_equal(a.grids, b.grids)
    np.testing.assert_array_equal(a.cells, b.cells)
    np.testing.assert_array_equal(a.density, b.density)
    np.testing.assert_array_equal(a.albedo_u8, b.albedo_u8)
    for up in (True, False):
        np.testing.assert_array_equal(a.neighbors(up), b.neighbors(up))


def points(levels, seed, n):
    """A lattice that is zero but for n points, many of them on borders."""
    L = 8 * 4 ** levels + 1
    rng = np.random.default_rng(seed)
    d = np.zeros((L, L, L), np.float32)
    edge = [0, 1, 7, 8, 9, L - 10, L - 9, L - 2, L - 1] + ([127, 128, 255, 256] if L > 129 else [])
    for _ in range(n):
        z, y, x = (int(rng.choice(edge)) if rng.random() < 0.6 else int(rng.integers(0, L))
                   for _ in range(3))
        d[z, y, x] = rng.choice([1.0, -0.5, 1e-8, 0.25])
    rgb = rng.integers(0, 256, (L, L, L, 3)).astype(np.uint8)
    return d, rgb


@pytest.mark.parametrize("levels,seed,n", [(1, 1, 1), (1, 2, 9), (1, 3, 200), (2, 4, 1), (2, 5, 40),
                                           (2, 6, 3000), (3, 7, 60)])
def test_border_points(yoxel_mod, levels, seed, n):
    import torch
    d, rgb = points(levels, seed, n)
    ref = yoxel_mod.BrickVolume.from_dense(levels, d, rgb)
    got = yoxel_mod.BrickVolume.build_dense(torch.from_numpy(d).cuda(), levels,
                                            torch.from_numpy(rgb).cuda())
    equal_volumes(got, ref)


@pytest.mark.parametrize("off_d,off_c", [(1, 0), (0, 1), (0, 2), (0, 3), (3, 1)])
@pytest.mark.parametrize("levels", [1, 2])
def test_unaligned_arrays(yoxel_mod, levels, off_d, off_c):
    """A lattice off_d floats and colours off_c bytes past an aligned address."""
    import torch
    d, rgb = points(levels, 20 + off_d + off_c, 500)
    ref = yoxel_mod.BrickVolume.from_dense(levels, d, rgb)
    bd = torch.zeros(d.size + 4, device="cuda")
    bc = torch.zeros(rgb.size + 4, dtype=torch.uint8, device="cuda")
    td = bd[off_d:off_d + d.size].view(d.shape)
    tc = bc[off_c:off_c + rgb.size].view(rgb.shape)
    td.copy_(torch.from_numpy(d))
    tc.copy_(torch.from_numpy(rgb))
    equal_volumes(yoxel_mod.BrickVolume.build_dense(td, levels, tc), ref)


@pytest.mark.parametrize("precision", [0, 1, 2, 3])
def test_device_neighbours(yoxel_mod, precision):
    """The apron fold of a device-built pool equals the upload's: the same
    neighbour tables."""
    import torch

    from yoxel import _lib as L
    d, rgb = points(2, 33, 900)
    vol = yoxel_mod.BrickVolume.from_dense(2, d, rgb)
    a = vol.upload(precision)
    b = yoxel_mod.VolumeGPU.from_dense(torch.from_numpy(d).cuda(), 2, precision,
                                       torch.from_numpy(rgb).cuda())
    g = torch.arange(vol.nbricks * 729, device="cuda", dtype=torch.float32) % 1021
    out = []
    for v in (a, b):
        t = g.clone()
        L.check(L.lib.yv_volume_fold_aprons(C.byref(v.desc()), C.c_void_p(t.data_ptr()), None,
                                            None), "fold")
        torch.cuda.synchronize()
        out.append(t)
    assert torch.equal(*out)
