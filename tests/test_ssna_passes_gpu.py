"""The count of blur passes that a frame launches, over cameras, voxel sizes and
widths, against the limits and the least depth of the unit cube in 64 bits."""
import numpy as np
import pytest

from conftest import camera_for
from oracle import ssna as O

pytestmark = pytest.mark.gpu


def renderer(yoxel_mod, dist, w, h, fov=60.0, **cam):
    r = yoxel_mod.Renderer()
    r.SetScene(yoxel_mod.SVOScene.spheres(5, 20, 2.0, 6.0, 5))
    pos, view = camera_for(dist=dist, **cam)
    r.SetViewPos(pos)
    r.SetViewDir(view)
    r.SetResolution(w, h)
    r.SetFOV(fov)
    return r, pos, view


@pytest.mark.parametrize("dist", [0.3, 1.5, 2.0, 6.0])
@pytest.mark.parametrize("w,h", [(64, 48), (640, 480), (1920, 1080)])
def test_passes_of_the_limits_that_reach_the_cube(yoxel_mod, dist, w, h):
    r, pos, view = renderer(yoxel_mod, dist, w, h)
    f = np.asarray(view, np.float64)
    f /= np.linalg.norm(f)
    corners = np.array([[x, y, z] for x in (0, 1) for y in (0, 1) for z in (0, 1)], np.float64)
    least = ((corners - np.asarray(pos, np.float64)) @ f).min()
    seen = set()
    p = r.ssna_params()
    for passes in (0, 1, 5, 64):
        for voxel in (1 / 16384, 1 / 2048, 1 / 256, 1 / 16, 4.0):
            p.blur_passes, p.voxel_size = passes, voxel
            n = r.ssna_passes(p)
            seen.add(n)
            z = [float(v) for v in O.zlimits(passes, voxel, 60.0, w)]
            # launched: every pass that reaches the cube; not launched: passes that
            # end more than a hundredth (of the depth and of a scene side) before it
            reach = sum(v >= least for v in z)
            near = sum(v >= least * (0.99 if least > 0 else 1.01) - 0.01 for v in z)
            assert reach <= n <= near
    assert len(seen) > 1
    p.ssna = 0
    assert r.ssna_passes(p) == 0


def test_refuses(yoxel_mod):
    r, _, _ = renderer(yoxel_mod, 1.5, 64, 48)
    p = r.ssna_params()
    for field, value in (("blur_passes", -1), ("blur_passes", 65), ("voxel_size", 0.0),
                         ("voxel_size", float("nan")), ("edge_threshold", -1.0)):
        q = r.ssna_params()
        setattr(q, field, value)
        with pytest.raises(Exception):
            r.ssna_passes(q)
        with pytest.raises(Exception):
            r.render_ssna(q)
    empty = yoxel_mod.Renderer()
    with pytest.raises(Exception):
        empty.ssna_passes(p)
