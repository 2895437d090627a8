"""Parameter arrays of the differentiable march that go on past the pool's points, or
end before them."""
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["albedo", "density", "both"])
def test_longer_arrays(yoxel_mod, which):
    """Albedo of more bricks than the density, density of more values a brick
    than a lattice has (the pool is its first values): the rest of them has no
    gradient, whatever the memory held."""
    import torch
    tv = yoxel_mod.BrickVolume.noise(1, 0.4, 1.4, 8).to_torch()
    nb = tv["density"].shape[0]
    cams = yoxel_mod.sphere_cameras(2)
    gen = torch.Generator(device="cuda").manual_seed(3)
    g = torch.randn((2, 24, 40, 4), generator=gen, device="cuda")

    def grads(den, alb):
        den.requires_grad_(True)
        alb.requires_grad_(True)
        rgba = yoxel_mod.volume_march(den, alb, tv, cams, 40, 24)
        # the memory the allocator hands out next is not zero
        for like in (den, alb):
            torch.full_like(like, 3e38)
        return torch.autograd.grad(rgba, (den, alb), g)

    ref = grads(tv["density"].clone(), tv["albedo"].clone())
    den, alb = tv["density"].clone(), tv["albedo"].clone()
    if which in ("albedo", "both"):
        alb = torch.cat([alb, torch.ones((nb,) + tuple(alb.shape[1:]), device="cuda")])
    if which in ("density", "both"):
        den = torch.cat([den.reshape(-1), torch.ones(nb * 729, device="cuda")]).view(nb, 2 * 729)
    got = grads(den, alb)
    for a, b in zip(got, ref):
        a, b = a.reshape(-1), b.reshape(-1)
        assert bool((a[b.numel():] == 0).all())
        # FP32 sums of the same terms in the order of the atomics: sqrt(256) 2^-24
        assert float((a[:b.numel()] - b).norm() / b.norm()) < 1e-6


def test_shorter_arrays_are_refused(yoxel_mod):
    """Refused before anything is allocated on a device or launched."""
    import torch
    nb = 3
    tv = dict(grids=torch.zeros((1, 64), dtype=torch.int32), levels=1,
              nbr_up=torch.zeros((nb, 7), dtype=torch.int32),
              nbr_dn=torch.zeros((nb, 7), dtype=torch.int32))
    den, alb = torch.zeros((nb, 729)), torch.zeros((nb, 729, 3))
    cams = yoxel_mod.sphere_cameras(1)
    for d, a in ((den[:, :-1].contiguous(), alb), (den, alb[:, :, :2].contiguous()),
                 (den, alb[:-1]), (den.half(), alb), (den, alb.half())):
        with pytest.raises(ValueError):
            yoxel_mod.volume_march(d, a, tv, cams, 8, 8)
        with pytest.raises(ValueError):
            yoxel_mod.pack_volume(d, a)


@pytest.mark.gpu
@pytest.mark.parametrize("table", ["nbr_up", "nbr_dn"])
def test_short_neighbour_tables_are_refused(yoxel_mod, table):
    import torch
    tv = yoxel_mod.BrickVolume.noise(1, 0.4, 1.4, 8).to_torch()
    cams = yoxel_mod.sphere_cameras(1)
    den = tv["density"].clone().requires_grad_(True)
    rgba = yoxel_mod.volume_march(den, tv["albedo"], {**tv, table: tv[table][:-1]}, cams, 16, 16)
    with pytest.raises(ValueError):
        torch.autograd.grad(rgba.sum(), den)
