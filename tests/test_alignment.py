"""Arrays that do not start where the kernels' wide loads and stores need them to:
refused before anything is launched (the pointers of these descriptors are never
followed), or taken through an aligned copy."""
import ctypes as C

import pytest

GOOD = 0x10000


def desc(L, precision, density=GOOD, albedo=GOOD):
    d = L.VolumeDevice()
    d.grids, d.ngrids, d.levels = GOOD, 1, 2
    d.density, d.albedo = density, albedo
    d.nbricks, d.precision = 8, precision
    d.nbr_up = d.nbr_dn = GOOD
    return d


def calls(L, d, rgba, grad):
    """Status of every call that marches d with these float4 frames."""
    lib, ok = L.lib, C.c_void_p(GOOD)
    cam = L.Camera(L.F3(0.5, 0.5, 3.0), L.F3(0.0, 0.0, -1.0), L.F3(0.0, 1.0, 0.0), 60.0)
    mp = C.byref(L.MarchParams(1.0, 0.5))
    r, g, ref = C.c_void_p(rgba), C.c_void_p(grad), C.byref(d)
    out = [lib.yv_volume_render(ref, cam, 1, 8, 8, mp, r, None, None, None),
           lib.yv_volume_render_tiles(ref, cam, 1, 8, 8, mp, 0, 1, r, None, None, None)]
    if d.precision in (1, 2):
        out += [lib.yv_volume_backward(ref, cam, 1, 8, 8, mp, r, g, ok, ok, None),
                lib.yv_volume_train_backward(ref, cam, 1, 8, 8, mp, r, g, ok, ok, None)]
    return out


@pytest.mark.parametrize("off", [1, 2, 4, 8, 12])
def test_pools(yoxel_mod, off):
    from yoxel import _lib as L
    size = {0: (2, 4), 1: (4, 4), 2: (None, 16), 3: (None, 8)}
    for precision, (dsize, asize) in size.items():
        if dsize and off % dsize:
            assert set(calls(L, desc(L, precision, density=GOOD + off), GOOD, GOOD)) == \
                {L.YV_ERR_INVALID_ARG}
        if off % asize:
            d = desc(L, precision, albedo=GOOD + off)
            assert set(calls(L, d, GOOD, GOOD)) == {L.YV_ERR_INVALID_ARG}
            cam = L.Camera(L.F3(0.5, 0.5, 3.0), L.F3(0.0, 0.0, -1.0), L.F3(0.0, 1.0, 0.0), 60.0)
            assert L.lib.yv_volume_render_rgba8(C.byref(d), cam, 1, 8, 8,
                                                C.byref(L.MarchParams(1.0, 0.5)),
                                                C.c_void_p(GOOD), None) == L.YV_ERR_INVALID_ARG


@pytest.mark.parametrize("off", [4, 8, 12])
def test_frames(yoxel_mod, off):
    from yoxel import _lib as L
    for precision in range(4):
        assert set(calls(L, desc(L, precision), GOOD + off, GOOD)) == {L.YV_ERR_INVALID_ARG}
    for precision in (1, 2):
        assert set(calls(L, desc(L, precision), GOOD, GOOD + off)[2:]) == {L.YV_ERR_INVALID_ARG}


@pytest.mark.parametrize("off", [1, 4])
def test_leaf_attributes(yoxel_mod, off):
    from yoxel import _lib as L
    cam = L.Camera(L.F3(0.5, 0.5, 3.0), L.F3(0.0, 0.0, -1.0), L.F3(0.0, 1.0, 0.0), 60.0)
    light = L.Light(L.F3(0.0, 0.0, 1.0), 0.1, 0.9, 0)
    assert L.lib.yv_render_svo_noalloc(
        C.c_void_p(GOOD), 1, 0, C.c_void_p(GOOD + off), 4, C.byref(cam), C.byref(light), 8, 8,
        C.byref(L.FrameOutputs()), None) == L.YV_ERR_INVALID_ARG


@pytest.mark.gpu  # (a batch takes a device when it is made)
def test_batch(yoxel_mod):
    from yoxel import _lib as L
    b = C.c_void_p()
    L.check(L.lib.yv_batch_create(C.byref(b)), "yv_batch_create")
    cam = L.Camera(L.F3(0.5, 0.5, 3.0), L.F3(0.0, 0.0, -1.0), L.F3(0.0, 1.0, 0.0), 60.0)
    mp = L.MarchParams(1.0, 0.5)
    for d, rgba in ((desc(L, 2, albedo=GOOD + 8), GOOD), (desc(L, 3, albedo=GOOD + 4), GOOD),
                    (desc(L, 0), GOOD + 4)):
        assert L.lib.yv_batch_add_volume(b, C.byref(d), C.byref(cam), 8, 8, C.byref(mp),
                                         C.c_void_p(rgba)) == L.YV_ERR_INVALID_ARG
    L.lib.yv_batch_destroy(b)


@pytest.mark.gpu
@pytest.mark.parametrize("off", [1, 2, 3])
def test_gradient_view(yoxel_mod, off):
    """A gradient of the frame that is a view starting inside a pixel."""
    import torch
    tv = yoxel_mod.BrickVolume.noise(1, 0.4, 1.4, 8).to_torch()
    cams = yoxel_mod.sphere_cameras(2)
    n = 2 * 24 * 40 * 4
    gen = torch.Generator(device="cuda").manual_seed(3)
    buf = torch.randn(n + 4, generator=gen, device="cuda")
    view = buf[off:off + n].view(2, 24, 40, 4)
    assert view.data_ptr() % 16 and view.is_contiguous()
    out = []
    for g in (view, view.clone()):
        den = tv["density"].clone().requires_grad_(True)
        alb = tv["albedo"].clone().requires_grad_(True)
        rgba = yoxel_mod.volume_march(den, alb, tv, cams, 40, 24)
        out.append(torch.autograd.grad(rgba, (den, alb), g))
    # FP32 sums of the same terms in the order of the atomics: sqrt(256) 2^-24
    for a, b in zip(*out):
        assert float(b.norm()) > 0 and float((a - b).norm() / b.norm()) < 1e-6
