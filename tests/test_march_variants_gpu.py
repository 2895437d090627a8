"""Variants of the brick march against each other: warps that march 8, 16 or 32
rays."""
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
