"""Batches that hold a pool with shared subtrees beside brick volumes, at each
register budget: the frames of separate launches."""
import pytest

from conftest import LIGHT, camera_for
from test_shared_pools_gpu import pool

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("budget", [0, 2, 3, 4])
@pytest.mark.parametrize("precisions", [(), (3,), (0, 2)])
def test_batch_equals_separate(yoxel_mod, budget, precisions):
    import torch
    w, h = 96, 72
    pos, view = camera_for()
    batch, outs, keep = yoxel_mod.Batch(), [], []
    spheres = yoxel_mod.SVOScene.spheres(5, 20, 2.0, 6.0, 5)
    for k in range(3):
        r = yoxel_mod.Renderer()
        if k == 1:
            r.SetScene(spheres)
        else:
            r.SetSceneArrays(*pool(8, 5 + 30 * k, 0.5, k))
        r.SetViewPos(pos)
        r.SetViewDir(view)
        r.SetResolution(w, h)
        r.SetFOV(60.0)
        r.SetLight(LIGHT, 0.15, 0.85, True)
        o = {n: torch.zeros((h, w), dtype=torch.int32, device="cuda") for n in ("rgba", "hit")}
        batch.add_svo(r, **o)
        outs += list(o.values())
        keep.append(r)
    for p in precisions:
        g = yoxel_mod.BrickVolume.noise(1, 0.4, 1.4, 8).upload(p)
        o = torch.zeros((h, w, 4), device="cuda")
        batch.add_volume(g.desc(), yoxel_mod.sphere_cameras(3)[1], w, h, o)
        outs.append(o)
        keep.append(g)
    batch.render_separate()
    torch.cuda.synchronize()
    ref = [o.clone() for o in outs]
    for o in outs:
        o.fill_(-1)
    batch.set_launch_config(blocks_per_sm=budget)
    for graph in (False, True):
        batch.render(graph=graph)
        torch.cuda.synchronize()
        for a, b in zip(outs, ref):
            assert torch.equal(a, b)
            assert len(torch.unique(b)) > 2
            a.fill_(-1)
