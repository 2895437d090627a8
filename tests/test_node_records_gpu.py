"""Node records on the device against the FP32 oracle where their numbering is
not that of a canonical pool: subtrees that several parents share, leaves that
share attributes, an odd number of records staged in shared memory."""
import numpy as np
import pytest

from conftest import LIGHT, camera_for

pytestmark = pytest.mark.gpu

EMPTY = 0x80000000


def _pool(kind, rng):
    """(nodes, root, attrs) of three node levels: every grandchild node of the
    root is one of `n` shared ones (kind "shared") or its own."""
    from yoxel import ATTR_DTYPE, NODE_DTYPE
    attrs = np.zeros(7, ATTR_DTYPE)
    attrs["rgb"][:, :3] = rng.integers(0, 256, (7, 3))
    attrs["n"][:, :3] = rng.integers(-127, 128, (7, 3))
    nodes = []

    def bottom():
        ch = np.full(8, EMPTY, np.uint32)
        fl = 0xFF00
        for c in range(8):
            if rng.random() < 0.5:
                ch[c] = rng.integers(0, 7)
                fl = (fl | (1 << c)) & ~(1 << (8 + c))
        nodes.append((fl, 0, ch))
        return len(nodes) - 1

    shared = [bottom() for _ in range(3)]

    def inner(children):
        ch = np.full(8, EMPTY, np.uint32)
        fl = 0xFF00
        for c in range(8):
            if rng.random() < 0.7:
                ch[c] = children()
                fl &= ~(1 << (8 + c))
        nodes.append((fl, 0, ch))
        return len(nodes) - 1

    pick = (lambda: int(rng.choice(shared))) if kind == "shared" else bottom
    mids = [inner(pick) for _ in range(3)]
    mid = (lambda: int(rng.choice(mids))) if kind == "shared" else (lambda: inner(pick))
    root = inner(mid)
    out = np.zeros(len(nodes), NODE_DTYPE)
    for i, (fl, d, ch) in enumerate(nodes):
        out[i]["flags"], out[i]["data"], out[i]["child"] = fl, d, ch
    return out, root, attrs


@pytest.mark.parametrize("kind", ["shared", "own"])
@pytest.mark.parametrize("staged", [0, 3])
def test_shared_nodes_and_attributes(oracle, yoxel_mod, kind, staged):
    nodes, root, attrs = _pool(kind, np.random.default_rng(11))
    pos, view = camera_for()
    w, h = 96, 64
    r = yoxel_mod.Renderer()
    r.SetSceneArrays(nodes, root, attrs)
    r.SetLaunchConfig(smem_nodes=staged)
    r.SetViewPos(pos)
    r.SetViewDir(view)
    r.SetResolution(w, h)
    r.SetFOV(60.0)
    r.SetLight(LIGHT, 0.15, 0.85, True)
    out = r.render_outputs()
    ref = oracle.svo_render(nodes.view(np.uint32).reshape(-1), root,
                            attrs.view(np.uint8).reshape(-1), pos, view, [0, 0, 1], 60.0, w, h,
                            LIGHT, shadows=True)
    assert out["stats"]["hits"] > 100
    for k in ("hit", "rgba", "fetches", "shadow_fetches"):
        np.testing.assert_array_equal(out[k].cpu().numpy().view(np.uint32).reshape(-1),
                                      np.asarray(ref[k], np.uint32).reshape(-1), err_msg=k)
    # the nodes reachable from the root, shared ones once
    seen, todo = set(), [root]
    while todo:
        i = todo.pop()
        if i in seen:
            continue
        seen.add(i)
        todo += [int(c) for k, c in enumerate(nodes[i]["child"])
                 if not (nodes[i]["flags"] >> k) & 1 and not c & EMPTY]
    assert r.device_scene_info()[0] == len(seen)


# frames around the sizes where a warp takes 8, 16 or 32 rays (from 8 rays a
# warp on 152 SMs x 3 blocks x 8 warps: 29184 and 58368 ray ids), partial tiles
@pytest.mark.parametrize("size", [(1, 1), (7, 3), (9, 5), (160, 120), (216, 136), (251, 233),
                                  (333, 175), (640, 95)])
@pytest.mark.parametrize("shadows", [False, True])
def test_small_frames(oracle, yoxel_mod, size, shadows):
    scene = yoxel_mod.SVOScene.spheres(6, 40, 2.0, 8.0, 77)
    pos, view = camera_for()
    w, h = size
    r = yoxel_mod.Renderer()
    r.SetScene(scene)
    r.SetViewPos(pos)
    r.SetViewDir(view)
    r.SetResolution(w, h)
    r.SetFOV(60.0)
    r.SetLight(LIGHT, 0.15, 0.85, shadows)
    out = r.render_outputs()
    ref = oracle.svo_render(scene.nodes_u32, scene.root, scene.attrs_u8, pos, view, [0, 0, 1],
                            60.0, w, h, LIGHT, shadows=shadows)
    for k in ("hit", "rgba", "fetches", "shadow_fetches"):
        np.testing.assert_array_equal(out[k].cpu().numpy().view(np.uint32), ref[k], err_msg=k)
    np.testing.assert_array_equal(out["hit_t"].cpu().numpy(), ref["hit_t"])
    assert out["stats"]["primary_rays"] == w * h
