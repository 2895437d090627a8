"""Brick pools with more lattice points than 32-bit point numbers reach are
refused before anything is launched: the pointers of these descriptors are never
followed."""
import ctypes as C

import pytest

# the first count whose 729 points a brick wrap, one whose points wrap to a few,
# and the largest count a descriptor holds
COUNTS = [2 ** 32 // 729 + 1, 2 ** 32 // 729 * 2 + 3, 2 ** 32 - 1]


def desc(L, n, precision):
    d = L.VolumeDevice()
    d.grids, d.ngrids, d.levels = 0x1000, 1, 4
    d.density, d.albedo = 0x1000, 0x1000
    d.nbricks, d.precision = n, precision
    d.nbr_up = d.nbr_dn = 0x1000
    return d


@pytest.mark.parametrize("n", COUNTS)
def test_calls_refuse(yoxel_mod, n):
    from yoxel import _lib as L
    lib, p = L.lib, C.c_void_p(0x1000)
    cam = L.Camera(L.F3(0.5, 0.5, 3.0), L.F3(0.0, 0.0, -1.0), L.F3(0.0, 1.0, 0.0), 60.0)
    mp = C.byref(L.MarchParams(1.0, 0.5))
    for precision in range(4):
        d = C.byref(desc(L, n, precision))
        assert lib.yv_volume_render(d, cam, 1, 8, 8, mp, p, None, None, None) == \
            L.YV_ERR_UNSUPPORTED
        assert lib.yv_volume_render_tiles(d, cam, 1, 8, 8, mp, 0, 1, p, None, None, None) == \
            L.YV_ERR_UNSUPPORTED
        assert lib.yv_volume_render_rgba8(d, cam, 1, 8, 8, mp, p, None) == L.YV_ERR_UNSUPPORTED
        assert lib.yv_volume_train_forward(d, p, p, cam, 1, 8, 8, mp, p, p, p, None) == \
            L.YV_ERR_UNSUPPORTED
    for precision in (1, 2):
        d = C.byref(desc(L, n, precision))
        assert lib.yv_volume_backward(d, cam, 1, 8, 8, mp, p, p, p, p, None) == \
            L.YV_ERR_UNSUPPORTED
        assert lib.yv_volume_train_backward(d, cam, 1, 8, 8, mp, p, p, p, p, None) == \
            L.YV_ERR_UNSUPPORTED
        assert lib.yv_volume_fold_aprons(d, p, p, None) == L.YV_ERR_UNSUPPORTED
        assert lib.yv_volume_sync_aprons(d, p, p, None) == L.YV_ERR_UNSUPPORTED


@pytest.mark.gpu  # (a batch takes a device when it is made)
@pytest.mark.parametrize("n", COUNTS)
def test_batch_refuses(yoxel_mod, n):
    from yoxel import _lib as L
    b = C.c_void_p()
    L.check(L.lib.yv_batch_create(C.byref(b)), "yv_batch_create")
    cam = L.Camera(L.F3(0.5, 0.5, 3.0), L.F3(0.0, 0.0, -1.0), L.F3(0.0, 1.0, 0.0), 60.0)
    mp = L.MarchParams(1.0, 0.5)
    for precision in range(4):
        assert L.lib.yv_batch_add_volume(b, C.byref(desc(L, n, precision)), C.byref(cam), 8, 8,
                                         C.byref(mp), C.c_void_p(0x1000)) == L.YV_ERR_UNSUPPORTED
    L.lib.yv_batch_destroy(b)


def test_pack_refuses(yoxel_mod):
    class Fake:  # a density whose shape is all that is looked at
        shape = (2 ** 32 // 729 + 1, 729)

    with pytest.raises(ValueError):
        yoxel_mod.pack_volume(Fake(), None)
