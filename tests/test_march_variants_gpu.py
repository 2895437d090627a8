"""Variants of the brick march against each other: warps that march 8, 16 or 32
rays, and the fitting step's forward (empty cells passed over) and backward
(gradients folded in one pass) against the plain entry points they stand for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def volume(yoxel_mod, levels, kind, seed=5):
    """A dense lattice as learnable tensors: "sparse" (most cells empty),
    "dense" (no empty cell) or "mixed" (half of the volume dense)."""
    import torch
    n = 8 * 4 ** levels + 1
    g = torch.Generator(device="cuda").manual_seed(seed)
    t = torch.rand((1, 1, 9, 9, 9), generator=g, device="cuda")
    d = torch.nn.functional.interpolate(t, size=(n, n, n), mode="trilinear",
                                        align_corners=True)[0, 0]
    if kind == "sparse":
        d = (d - 0.6).clamp_(min=0.0)
    elif kind == "mixed":
        d[:, :, : n // 2] = (d[:, :, : n // 2] - 0.6).clamp_(min=0.0)
    rgb = (torch.rand((n, n, n, 3), generator=g, device="cuda") * 255).to(torch.uint8)
    return yoxel_mod.BrickVolume.build_dense(d.contiguous(), levels, rgb).to_torch()


# 152 SMs x 24 warps: a launch of up to 912 tiles of 8x4 pixels marches 8 rays
# a warp, up to 1824 16, above that 32 (tiles of whole 16x16 squares)
@pytest.mark.parametrize("size", [(1, 1), (5, 3), (17, 9), (64, 64), (181, 161), (241, 239),
                                  (250, 246)])
def test_small_launches_equal_large_ones(yoxel_mod, size):
    import torch
    tv = volume(yoxel_mod, 1, "sparse")
    w, h = size
    desc = yoxel_mod.torch_desc(tv)
    cams = yoxel_mod.sphere_cameras(40)
    many = yoxel_mod.render_volume(desc, cams, w, h)
    for k in (0, 17):
        one = yoxel_mod.render_volume(desc, [cams[k]], w, h)
        assert torch.equal(one[0], many[k])
    if w * h >= 4096:  # (a frame of few pixels has its corner rays only)
        assert float(many.abs().sum()) > 0


@pytest.mark.parametrize("kind", ["sparse", "mixed", "dense"])
@pytest.mark.parametrize("levels", [1, 2])
def test_fitting_forward_equals_plain_march(yoxel_mod, kind, levels):
    import torch
    tv = volume(yoxel_mod, levels, kind)
    cams = yoxel_mod.sphere_cameras(3)
    got = yoxel_mod.volume_march(tv["density"], tv["albedo"], tv, cams, 93, 61, 1.5, 0.5)
    packed = yoxel_mod.pack_volume(tv["density"], tv["albedo"])
    ref = yoxel_mod.render_volume(yoxel_mod.torch_desc(tv, packed=packed), cams, 93, 61, 1.5, 0.5)
    assert torch.equal(got, ref)
    assert float(ref[..., 3].max()) > 0.5


def test_not_finite_values_reach_the_frame(yoxel_mod):
    """NaN and infinity in the parameters show where the plain march shows
    them, also in cells whose densities are all zero."""
    import torch
    tv = volume(yoxel_mod, 1, "sparse")
    den, alb = tv["density"].clone(), tv["albedo"].clone()
    empty = (den == 0).nonzero()
    for i, v in enumerate((float("nan"), float("inf"), float("-inf"))):
        b, p = empty[(i + 1) * len(empty) // 5].tolist()
        alb[b, p, i] = v
    b, p = (den > 0).nonzero()[7].tolist()
    den[b, p] = float("nan")
    cams = yoxel_mod.sphere_cameras(6)
    got = yoxel_mod.volume_march(den, alb, tv, cams, 64, 64)
    packed = yoxel_mod.pack_volume(den, alb)
    ref = yoxel_mod.render_volume(yoxel_mod.torch_desc(tv, packed=packed), cams, 64, 64)
    assert bool(ref.isnan().any())
    assert torch.equal(got.nan_to_num(nan=-7.0), ref.nan_to_num(nan=-7.0))


@pytest.mark.parametrize("kind", ["sparse", "dense"])
@pytest.mark.parametrize("size", [(16, 16), (250, 246)])
def test_fitting_backward_equals_backward_and_fold(yoxel_mod, kind, size):
    import torch
    tv = volume(yoxel_mod, 1, kind)
    den = tv["density"].clone().requires_grad_(True)
    alb = tv["albedo"].clone().requires_grad_(True)
    cams = yoxel_mod.sphere_cameras(2)
    w, h = size
    rgba = yoxel_mod.volume_march(den, alb, tv, cams, w, h)
    g = torch.from_numpy(np.random.default_rng(3).standard_normal(rgba.shape).astype(np.float32))
    g = g.cuda()
    gd, ga = torch.autograd.grad(rgba, (den, alb), g)
    packed = yoxel_mod.pack_volume(den.detach(), alb.detach())
    rd, ra = torch.zeros_like(gd), torch.zeros_like(ga)
    yoxel_mod.volume_backward(yoxel_mod.torch_desc(tv, packed=packed), cams, w, h, rgba.detach(),
                              g, rd, ra)
    # FP32 sums of the same terms in another order (atomics): up to some
    # thousand per point, sqrt(4096) 2^-24 = 4e-6
    for a, b in ((gd, rd), (ga, ra)):
        assert float((a - b).norm() / b.norm()) < 4e-6
    # far-side copies equal their owners, 0 where there is none
    up = tv["nbr_up"].cpu().numpy()
    v = gd.cpu().numpy().reshape(-1, 9, 9, 9)
    for b in range(len(v)):
        own = v[up[b, 0], :8, :8, 0] if up[b, 0] >= 0 else 0.0
        assert np.array_equal(v[b, :8, :8, 8], np.broadcast_to(own, (8, 8)))


@pytest.mark.parametrize("precision", [0, 1, 2, 3])
def test_register_budgets_agree(yoxel_mod, precision):
    """A launch whose warps all fit at the small register budget, and one that
    does not, of every lattice format."""
    import torch
    gv = yoxel_mod.BrickVolume.noise(1, 0.4, 1.4, 8).upload(precision)
    cams = yoxel_mod.sphere_cameras(50)
    many = yoxel_mod.render_volume(gv.desc(), cams, 67, 43)
    for k in (0, 31):
        assert torch.equal(yoxel_mod.render_volume(gv.desc(), [cams[k]], 67, 43)[0], many[k])
    assert float(many[..., 3].max()) > 0.1


@pytest.mark.parametrize("special", [None, float("inf"), float("nan")])
def test_gradient_scratch_layouts_agree(yoxel_mod, special):
    """64 frames keep edge records in the gradient scratch, one frame points;
    the other 63 frames have no gradient."""
    import torch
    tv = volume(yoxel_mod, 1, "sparse")
    cam = yoxel_mod.sphere_cameras(5)[2]
    rng = np.random.default_rng(4)
    one = torch.from_numpy(rng.standard_normal((1, 40, 40, 4)).astype(np.float32)).cuda()
    if special is not None:
        one[0, 17, 21, 1] = special
    many = torch.zeros((64, 40, 40, 4), device="cuda")
    many[0] = one[0]
    out = []
    for cams, g in (([cam], one), ([cam] * 64, many)):
        den = tv["density"].clone().requires_grad_(True)
        alb = tv["albedo"].clone().requires_grad_(True)
        rgba = yoxel_mod.volume_march(den, alb, tv, cams, 40, 40)
        out.append(torch.autograd.grad(rgba, (den, alb), g))
    for a, b in zip(*out):
        assert torch.equal(a.isfinite(), b.isfinite())
        a, b = a.nan_to_num(0.0, 0.0, 0.0), b.nan_to_num(0.0, 0.0, 0.0)
        # FP32 sums of at most some hundred terms per point in another order:
        # sqrt(256) 2^-24 = 1e-6
        assert float((a - b).norm() / b.norm()) < 1e-6
        assert float(b.norm()) > 0
