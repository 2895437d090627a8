"""SSNA blur passes at the edge of the launch rule: a pass whose limit lies
below every depth the unit cube can have is not launched.

A solid cube seen face on from a known distance: the smallest hit depth is the
face's, which is also the least depth the cube allows, so a pass limit placed
a little below, at and above it is at the rule's edge.  Bar: blurred depth and
normals bit-exact with the FP32 numpy restatement, which runs every pass."""
import numpy as np
import pytest

from conftest import LIGHT
from oracle import ssna as O

pytestmark = pytest.mark.gpu

W, H = 72, 48


@pytest.fixture(scope="module")
def cube(yoxel_mod):
    n = 32
    field = np.ones((n, n, n), np.float32)
    # steps in the face, so that blurring changes depths
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    rough = ((i * 7 + j * 3) % 5) == 0
    field[:, :, -1][rough] = 0.0
    field[-1][rough] = 0.0
    field[:, -1][rough] = 0.0
    return field


@pytest.mark.parametrize("fov", [25.0, 60.0, 170.0])
@pytest.mark.parametrize("dist", [0.02, 0.9, 40.0])
@pytest.mark.parametrize("rel", [-0.02, -1.0 / 128, -0.001, 0.0, 0.002, 0.3])
def test_limits_about_the_nearest_depth(yoxel_mod, cube, fov, dist, rel):
    import torch
    dev = torch.device("cuda", 0)
    scene = yoxel_mod.SVOScene.build_dense(torch.from_numpy(cube).to(dev), 5)
    r = yoxel_mod.Renderer()
    r.SetScene(scene)
    pos = np.array([1.0 + dist, 0.47, 0.53], np.float32)
    r.SetViewPos(pos)
    r.SetViewDir([-1, 0, 0])
    r.SetViewUp([0, 0, 1])
    r.SetResolution(W, H)
    r.SetFOV(fov)
    r.SetLight(LIGHT, 1.0, 0.0, False)
    tr = dict(rgba=torch.empty((H, W), dtype=torch.int32, device=dev),
              hit_t=torch.empty((H, W), dtype=torch.float32, device=dev),
              normal=torch.empty((H, W, 3), dtype=torch.float32, device=dev))
    r.render_async(**tr)
    r.frame_stats()
    tr = {k: v.cpu().numpy() for k, v in tr.items()}
    tr["rgba"] = tr["rgba"].view(np.uint32)
    hits = (tr["rgba"] >> 24) != 0
    assert hits.any()
    d0, du, dv = r.ray_basis()
    zmin = float(O.depth(tr["rgba"], tr["hit_t"], d0, du, dv)[hits].min())

    p = r.ssna_params()
    p.blur_passes = 4
    # the third pass has its limit at zmin (1 + rel)
    base = O.zlimits(4, 1.0, float(np.float32(fov)), W)[2]
    p.voxel_size = zmin * (1.0 + rel) / float(base)
    p.edge_threshold = 0.1
    dep = torch.empty((H, W), dtype=torch.float32, device=dev)
    nrm = torch.empty((H, W, 3), dtype=torch.float32, device=dev)
    r.render_ssna(p, depth=dep, normals=nrm)
    r.frame_stats()
    lights = [dict(pos=list(lt.pos), diffuse=list(lt.diffuse), specular=list(lt.specular),
                   attenuation=list(lt.attenuation)) for lt in p.lights if lt.enabled]
    _, o_dep, o_n = O.ssna_frame(tr["rgba"], tr["hit_t"], tr["normal"], pos, d0, du, dv,
                                 float(np.float32(fov)), passes=p.blur_passes,
                                 voxel_size=p.voxel_size, edge_threshold=p.edge_threshold,
                                 edge_pad=p.edge_pad, ssna=True, show_normals=False,
                                 ambient=list(p.ambient), specular_exp=p.specular_exp,
                                 lights=lights)
    assert np.array_equal(dep.cpu().numpy().view(np.uint32), o_dep.view(np.uint32))
    assert np.array_equal(nrm.cpu().numpy().view(np.uint32), o_n.view(np.uint32))
