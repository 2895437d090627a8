"""Frames with the level-of-detail cut-off at each register budget they can get
(by their size, or as the launch configuration asks): bit-exact with the FP32
oracle."""
import numpy as np
import pytest

from conftest import LIGHT, camera_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(yoxel_mod):
    return yoxel_mod.SVOScene.spheres(7, 60, 4.0, 24.0, 9).build_lod()


@pytest.mark.parametrize("blocks", [0, 2, 3, 4, 5])
@pytest.mark.parametrize("w,h", [(1, 1), (133, 67), (641, 479)])
def test_lod_frame_at_each_budget(yoxel_mod, oracle, scene, blocks, w, h):
    r = yoxel_mod.Renderer()
    r.SetScene(scene)
    pos, view = camera_for(dist=1.3)
    r.SetViewPos(pos)
    r.SetViewDir(view)
    r.SetViewUp([0, 0, 1])
    r.SetResolution(w, h)
    r.SetFOV(60.0)
    r.SetLight(LIGHT, 0.15, 0.85, True)
    r.SetDetailCoef(3.0)
    r.SetLaunchConfig(blocks_per_sm=blocks)
    g = r.render_outputs()
    o = oracle.svo_render(scene.nodes_u32, scene.root, scene.attrs_u8, pos, view,
                          np.float32([0, 0, 1]), 60.0, w, h, LIGHT, 0.15, 0.85, True,
                          lod_coef=r.lod_coef())
    for k in ("hit", "hit_t", "rgba", "fetches", "shadow_fetches"):
        a, b = g[k].cpu().numpy(), np.asarray(o[k])
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), k
