"""Where the backward changes the layout of its gradient scratch: gradients on both
sides of each line against the sum of one-camera backwards, which are too small
for edge records."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def volume(yoxel_mod, levels, bricks=None):
    """Smooth density with empty cells; bricks: about so many of them occupied."""
    import torch
    n = 8 * 4 ** levels + 1
    g = torch.Generator(device="cuda").manual_seed(5)
    t = torch.rand((1, 1, 17, 17, 17), generator=g, device="cuda")
    d = torch.nn.functional.interpolate(t, size=(n, n, n), mode="trilinear",
                                        align_corners=True)[0, 0]
    d = (d - 0.5).clamp_(min=0.0)
    if bricks:
        side = round(bricks ** (1 / 3))
        keep = torch.zeros_like(d)
        lo = (n - 1 - 8 * side) // 16 * 8
        keep[lo + 1:lo + 8 * side, lo + 1:lo + 8 * side, lo + 1:lo + 8 * side] = 1.0
        d = (d + 0.01) * keep
    rgb = (torch.rand((n, n, n, 3), generator=g, device="cuda") * 255).to(torch.uint8)
    return yoxel_mod.BrickVolume.build_dense(d.contiguous(), levels, rgb).to_torch()


# rays per lattice point below and above one in six (64 frames, 4096 bricks at
# most); 65 frames: a last launch of one, in the layout of the first; a pool on
# either side of 128 MB of edge records (17^3 and 18^3 bricks)
@pytest.mark.parametrize("levels,bricks,cams,size", [
    (2, None, 64, (80, 80)), (2, None, 64, (96, 96)), (1, None, 65, (64, 40)),
    (3, 17 ** 3, 64, (128, 96)), (3, 18 ** 3, 64, (128, 96))])
def test_layouts_agree_with_single_frames(yoxel_mod, levels, bricks, cams, size):
    import torch
    tv = volume(yoxel_mod, levels, bricks)
    if bricks:
        assert tv["density"].shape[0] == bricks
    w, h = size
    cs = yoxel_mod.sphere_cameras(cams)
    den = tv["density"].clone().requires_grad_(True)
    alb = tv["albedo"].clone().requires_grad_(True)
    rgba = yoxel_mod.volume_march(den, alb, tv, cs, w, h)
    rng = np.random.default_rng(3)
    g = torch.from_numpy(rng.standard_normal(tuple(rgba.shape)).astype(np.float32)).cuda()
    gd, ga = torch.autograd.grad(rgba, (den, alb), g)
    packed = yoxel_mod.pack_volume(den.detach(), alb.detach())
    desc = yoxel_mod.torch_desc(tv, packed=packed)
    rd, ra = torch.zeros_like(gd), torch.zeros_like(ga)
    frames = rgba.detach()
    for k in range(cams):
        yoxel_mod.volume_backward(desc, [cs[k]], w, h, frames[k], g[k], rd, ra, fold=k == cams - 1)
    # FP32 sums of the same terms in another order (atomics, and one frame after
    # another): up to some thousand per point, sqrt(4096) 2^-24 = 4e-6
    for a, b in ((gd, rd), (ga, ra)):
        assert float(b.norm()) > 0
        assert float((a - b).norm() / b.norm()) < 4e-6


# an unpacked fp32 pool in a launch that fills the GPU, and one that does not
@pytest.mark.parametrize("cams", [2, 64])
def test_unpacked_pool(yoxel_mod, cams):
    import torch
    tv = volume(yoxel_mod, 1)
    cs = yoxel_mod.sphere_cameras(cams)
    w, h = 64, 40
    plain = yoxel_mod.torch_desc(tv)
    packed_pool = yoxel_mod.pack_volume(tv["density"], tv["albedo"])
    packed = yoxel_mod.torch_desc(tv, packed=packed_pool)
    rgba = yoxel_mod.render_volume(plain, cs, w, h)
    assert torch.equal(rgba, yoxel_mod.render_volume(packed, cs, w, h))
    rng = np.random.default_rng(3)
    g = torch.from_numpy(rng.standard_normal(tuple(rgba.shape)).astype(np.float32)).cuda()
    out = []
    for desc in (plain, packed):
        # added to what the tensors hold
        gd, ga = torch.full_like(tv["density"], 0.5), torch.full_like(tv["albedo"], -0.25)
        yoxel_mod.volume_backward(desc, cs, w, h, rgba, g, gd, ga, fold=False)
        out.append((gd - 0.5, ga + 0.25))
    for a, b in zip(*out):
        # the same terms in the order of the atomics (4e-6, as above), and one
        # rounding to the spacing of 0.5 + gradient, 2^-24 of each value and of
        # 0.5, on either side
        bar = 4e-6 * float(b.norm()) + 2 * 2.0 ** -24 * float((b.abs() + 0.5).norm())
        assert float(b.norm()) > 0 and float((a - b).norm()) < bar
