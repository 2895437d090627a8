"""Frames with the first node records staged in shared memory, where the block's
shared memory passes 48 KB (32 KB of it the ring): the frame without staging."""
import pytest

from conftest import LIGHT, camera_for

pytestmark = pytest.mark.gpu


# 8 bytes a record: 2048 fill 16 KB; counts about it and about 512 (16 KB of
# 32-byte records), the cap of 4096 and beyond
@pytest.mark.parametrize("nodes", [1, 511, 512, 513, 2040, 2045, 2046, 2047, 2048, 2049, 2050,
                                   4095, 4096, 100000])
@pytest.mark.parametrize("threads", [0, 64])
def test_staged_counts(yoxel_mod, nodes, threads):
    import torch
    scene = yoxel_mod.SVOScene.spheres(7, 120, 3.0, 12.0, 77)
    assert scene.node_count > 4096
    pos, view = camera_for()
    r = yoxel_mod.Renderer()
    r.SetScene(scene)
    r.SetViewPos(pos)
    r.SetViewDir(view)
    r.SetResolution(200, 120)
    r.SetFOV(60.0)
    r.SetLight(LIGHT, 0.15, 0.85, True)
    ref = r.render_outputs()
    assert ref["stats"]["hits"] > 100
    for budget in (2, 3, 4, 5):
        r.SetLaunchConfig(smem_nodes=nodes, block_threads=threads, blocks_per_sm=budget)
        out = r.render_outputs()
        for k in ("rgba", "hit", "hit_t", "fetches", "shadow_fetches"):
            assert torch.equal(out[k], ref[k]), (budget, k)
