"""The two calls of a fitting step: their argument errors, and streams other than
the default one."""
import ctypes as C

import pytest

GOOD = 0x10000


def args(L):
    d = L.VolumeDevice()
    d.grids, d.ngrids, d.levels = GOOD, 1, 2
    d.albedo, d.nbricks, d.precision = GOOD, 8, 2
    d.nbr_up = d.nbr_dn = GOOD
    cam = L.Camera(L.F3(0.5, 0.5, 3.0), L.F3(0.0, 0.0, -1.0), L.F3(0.0, 1.0, 0.0), 60.0)
    return d, cam, L.MarchParams(1.0, 0.5)


def test_argument_errors(yoxel_mod):
    """Nothing is launched: the pointers are never followed."""
    from yoxel import _lib as L
    lib, p = L.lib, C.c_void_p(GOOD)

    def forward(d, cam, mp, density=p, albedo=p, n=1, w=8, h=8, packed=p, mask=p, rgba=p):
        return lib.yv_volume_train_forward(
            None if d is None else C.byref(d), density, albedo, cam, n, w, h,
            None if mp is None else C.byref(mp), packed, mask, rgba, None)

    def backward(d, cam, mp, rgba=p, grad=p, gd=p, ga=p, n=1, w=8, h=8):
        return lib.yv_volume_train_backward(
            None if d is None else C.byref(d), cam, n, w, h,
            None if mp is None else C.byref(mp), rgba, grad, gd, ga, None)

    d, cam, mp = args(L)
    bad = L.YV_ERR_INVALID_ARG
    for kw in (dict(density=None), dict(albedo=None), dict(packed=None), dict(mask=None),
               dict(rgba=None), dict(packed=C.c_void_p(GOOD + 8)), dict(n=0), dict(w=0),
               dict(h=-1)):
        assert forward(d, cam, mp, **kw) == bad, kw
    for kw in (dict(rgba=None), dict(grad=None), dict(gd=None), dict(ga=None), dict(n=0),
               dict(w=0)):
        assert backward(d, cam, mp, **kw) == bad, kw
    for call in (forward, backward):
        assert call(None, cam, mp) == bad
        assert call(d, None, mp) == bad
        assert call(d, cam, None) == bad
        assert call(d, cam, L.MarchParams(1.0, 0.0)) == bad
        assert call(d, cam, L.MarchParams(float("nan"), 0.5)) == bad
        wide = args(L)[1]
        wide.fov_deg = 180.0
        assert call(d, wide, mp) == bad
        away = args(L)[1]
        away.pos[0] = float("inf")
        assert call(d, away, mp) == bad
    for field in ("nbr_up", "nbr_dn"):
        e = args(L)[0]
        setattr(e, field, None)
        assert backward(e, cam, mp) == bad
    for precision in (0, 3):  # formats that have no adjoint
        e = args(L)[0]
        e.precision = precision
        e.density = GOOD
        assert backward(e, cam, mp) == bad
    e = args(L)[0]
    e.grids = None
    assert forward(e, cam, mp) == bad and backward(e, cam, mp) == bad


@pytest.mark.gpu
def test_side_streams(yoxel_mod):
    """Steps of two volumes, each on a stream of its own, interleaved: the frames
    and gradients of the default stream."""
    import torch
    cams = yoxel_mod.sphere_cameras(6)
    tvs = [yoxel_mod.BrickVolume.noise(1, 0.4 - 0.1 * k, 1.4, 8 + k).to_torch() for k in range(2)]
    params = [[tv[k].clone().requires_grad_(True) for k in ("density", "albedo")] for tv in tvs]
    gen = torch.Generator(device="cuda").manual_seed(4)
    g = torch.randn((6, 96, 96, 4), generator=gen, device="cuda")

    def step(i):
        rgba = yoxel_mod.volume_march(*params[i], tvs[i], cams, 96, 96)
        return (rgba.detach(),) + torch.autograd.grad(rgba, params[i], g)

    ref = [step(i) for i in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = [[], []]
    torch.cuda.synchronize()
    for _ in range(4):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(step(i))
    torch.cuda.synchronize()
    for i in range(2):
        for frame, gd, ga in got[i]:
            assert torch.equal(frame, ref[i][0])
            # FP32 sums of some thousand terms in the order of the atomics
            for a, b in ((gd, ref[i][1]), (ga, ref[i][2])):
                assert float((a - b).norm() / b.norm()) < 4e-6
