"""GPU SVO build where its level arrays have edges: levels of less than a word (depth
1 and 2), a grid whose levels above the bottom take several folds and whose prefix
sums carry over rounds of 1024 chunks (depth 10) - the pool against the CPU oracle
of the build, and the frame of the renderer's own records against the frame of the
oracle's pool."""
import numpy as np
import pytest

from conftest import LIGHT, camera_for

pytestmark = pytest.mark.gpu


def fields():
    out = []
    for depth in (1, 2, 3):
        for seed, share in ((1, 0.5), (2, 0.1), (3, 0.95)):
            out.append((depth, seed, share))
    return out


def grid(depth, seed, share):
    G = 1 << depth
    rng = np.random.default_rng(seed + 10 * depth)
    d = (share - rng.random((G, G, G))).astype(np.float32)
    rgb = rng.integers(0, 256, (G, G, G, 3), dtype=np.uint8)
    return d, rgb


def sparse_grid(depth):
    """Empty but for boxes: on the grid's corners and faces, one that a level's
    array is full of in its middle, single voxels, noise."""
    G = 1 << depth
    rng = np.random.default_rng(depth)
    d = np.zeros((G, G, G), np.float32)
    d[:3, :5, :2] = 1.0
    d[-1, -1, -1] = 0.5
    d[-9:, :7, -5:] = 1.0
    q = G // 4
    d[q:q + 70, q:q + 66, q:q + 40] = 2.0
    d[G // 2 - 9:G // 2 + 9, 3 * q:3 * q + 64, 3 * q - 20:3 * q + 20] = \
        rng.standard_normal((18, 64, 40)).astype(np.float32)
    for _ in range(200):
        x, y, z = rng.integers(0, G, 3)
        d[z, y, x] = 1.0
    return d


def renderer(yoxel_mod, w, h):
    pos, view = camera_for()
    r = yoxel_mod.Renderer()
    r.SetViewPos(pos)
    r.SetViewDir(view)
    r.SetResolution(w, h)
    r.SetFOV(60.0)
    r.SetLight(LIGHT, 0.15, 0.85, True)
    return r


def check(yoxel_mod, oracle, d, rgb, depth, w, h):
    import torch
    nodes, attrs, root = oracle.svo_build_dense(d, depth, 0.25, rgb)
    td = torch.from_numpy(d).cuda()
    tr = None if rgb is None else torch.from_numpy(rgb).cuda()
    s = yoxel_mod.SVOScene.build_dense(td, depth, 0.25, tr)
    assert s.root == root
    assert np.array_equal(s.nodes_u32.reshape(-1, 10), nodes)
    assert np.array_equal(s.attrs_u8.reshape(-1, 8), attrs)
    r = renderer(yoxel_mod, w, h)
    r.SetSceneDense(td, depth, 0.25, tr)
    got = r.render_outputs()
    pos, view = camera_for()
    ref = oracle.svo_render(nodes.reshape(-1), root, attrs.reshape(-1), pos, view,
                            np.float32([0, 0, 1]), 60.0, w, h, LIGHT, 0.15, 0.85, True)
    for k in ("hit", "rgba", "fetches", "shadow_fetches"):
        np.testing.assert_array_equal(got[k].cpu().numpy().view(np.uint32).reshape(-1),
                                      np.asarray(ref[k], np.uint32).reshape(-1), err_msg=k)
    return len(nodes), got["stats"]["hits"]


@pytest.mark.parametrize("depth,seed,share", fields())
def test_shallow(yoxel_mod, oracle, depth, seed, share):
    d, rgb = grid(depth, seed, share)
    n, hits = check(yoxel_mod, oracle, d, rgb, depth, 96, 64)
    assert (n > 0) == bool((d > 0.25).any()) and (hits > 100 or n == 0 or share < 0.5)


@pytest.mark.parametrize("depth", [9, 10])
def test_deep_and_sparse(yoxel_mod, oracle, depth):
    n, hits = check(yoxel_mod, oracle, sparse_grid(depth), None, depth, 320, 200)
    assert n > 1000 and hits > 100
