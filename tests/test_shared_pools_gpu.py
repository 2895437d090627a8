"""Pools whose subtrees have many parents (directed acyclic graphs): the memory of
their device records, and every kind of frame against the FP32 oracle."""
import numpy as np
import pytest

from conftest import LIGHT, camera_for

pytestmark = pytest.mark.gpu

EMPTY = 0x80000000


def pool(levels, per_level, fill, seed, attrs=9):
    """(nodes, root, attrs): `levels` levels of per_level nodes whose children are
    drawn from the level below, the root on top.  per_level 0: no node is shared."""
    from yoxel import ATTR_DTYPE, NODE_DTYPE
    rng = np.random.default_rng(seed)
    at = np.zeros(attrs, ATTR_DTYPE)
    at["rgb"][:, :3] = rng.integers(0, 256, (attrs, 3))
    at["n"][:, :3] = rng.integers(-127, 128, (attrs, 3))
    nodes = []

    def node(child):
        ch, fl = np.full(8, EMPTY, np.uint32), 0xFF00
        for c in range(8):
            if rng.random() < fill:
                if child is None:
                    ch[c] = rng.integers(0, attrs)
                    fl = (fl | (1 << c)) & ~(1 << (8 + c))
                else:
                    ch[c] = child()
                    fl &= ~(1 << (8 + c))
        nodes.append((fl, 0, ch))
        return len(nodes) - 1

    def tree(depth):
        return node(None if depth == 1 else lambda: tree(depth - 1))

    if per_level:
        below = [node(None) for _ in range(per_level)]
        for _ in range(levels - 2):
            below = [node(lambda b=below: int(rng.choice(b))) for _ in range(per_level)]
        root = node(lambda: int(rng.choice(below)))
    else:
        root = tree(levels)
    out = np.zeros(len(nodes), NODE_DTYPE)
    for i, (fl, d, ch) in enumerate(nodes):
        out[i]["flags"], out[i]["data"], out[i]["child"] = fl, d, ch
    return out, root, at


def counts(nodes, root):
    """(nodes reachable from the root, their node children, their leaves)."""
    seen, todo, edges, leaves = {root}, [root], 0, 0
    while todo:
        n = nodes[todo.pop()]
        for c in range(8):
            w = int(n["child"][c])
            if (n["flags"] >> c) & 1:
                leaves += 1
            elif not w & EMPTY:
                edges += 1
                if w not in seen:
                    seen.add(w)
                    todo.append(w)
    return len(seen), edges, leaves


def renderer(yoxel_mod, w, h, shadows=True):
    pos, view = camera_for()
    r = yoxel_mod.Renderer()
    r.SetViewPos(pos)
    r.SetViewDir(view)
    r.SetResolution(w, h)
    r.SetFOV(60.0)
    r.SetLight(LIGHT, 0.15, 0.85, shadows)
    return r


def oracle_frame(oracle, nodes, root, attrs, w, h, **kw):
    pos, view = camera_for()
    return oracle.svo_render(nodes.view(np.uint32).reshape(-1), root,
                             attrs.view(np.uint8).reshape(-1), pos, view,
                             np.float32([0, 0, 1]), 60.0, w, h, LIGHT, 0.15, 0.85, True, **kw)


def assert_same(out, ref):
    for k in ("hit", "rgba", "fetches", "shadow_fetches"):
        np.testing.assert_array_equal(out[k].cpu().numpy().view(np.uint32).reshape(-1),
                                      np.asarray(ref[k], np.uint32).reshape(-1), err_msg=k)
    np.testing.assert_array_equal(out["hit_t"].cpu().numpy().reshape(-1),
                                  np.asarray(ref["hit_t"]).reshape(-1))


# one node a level with all 8 children, few, many (each with one or two parents)
POOLS = [(5, 1, 1.0), (7, 3, 0.55), (9, 40, 0.5), (4, 700, 0.3), (6, 0, 0.5)]


@pytest.mark.parametrize("levels,per_level,fill", POOLS)
def test_memory(yoxel_mod, levels, per_level, fill):
    """No more than 16 bytes a node, 4 a node child and 4 a leaf, whatever the
    sharing; without any, no more than the nodes and leaves."""
    nodes, root, attrs = pool(levels, per_level, fill, 3)
    n, edges, leaves = counts(nodes, root)
    r = renderer(yoxel_mod, 16, 16)
    r.SetSceneArrays(nodes, root, attrs)
    got_nodes, got_bytes = r.device_scene_info()
    assert got_nodes == n
    assert got_bytes <= 16 * n + 4 * (edges if edges + 1 != n else 0) + 4 * leaves + 16 * len(attrs)


@pytest.mark.parametrize("levels,per_level,fill", POOLS)
@pytest.mark.parametrize("cfg", [dict(), dict(smem_nodes=5), dict(blocks_per_sm=2)])
def test_frames(oracle, yoxel_mod, levels, per_level, fill, cfg):
    nodes, root, attrs = pool(levels, per_level, fill, 5)
    w, h = 120, 88
    r = renderer(yoxel_mod, w, h)
    r.SetLaunchConfig(**cfg)
    r.SetSceneArrays(nodes, root, attrs)
    out = r.render_outputs()
    assert out["stats"]["hits"] > 100
    assert_same(out, oracle_frame(oracle, nodes, root, attrs, w, h))
    # another scene in the same renderer, then this one again
    other = yoxel_mod.SVOScene.spheres(5, 20, 2.0, 6.0, 5)
    r.SetScene(other)
    assert_same(r.render_outputs(), oracle_frame(oracle, other.nodes, other.root, other.attrs,
                                                 w, h))
    r.SetSceneArrays(nodes, root, attrs)
    assert_same(r.render_outputs(), oracle_frame(oracle, nodes, root, attrs, w, h))


@pytest.mark.parametrize("detail", [1.0, 6.0])
def test_detail_cut_off(oracle, yoxel_mod, detail):
    nodes, root, attrs = pool(9, 40, 0.5, 7)
    scene = yoxel_mod.SVOScene.from_arrays(nodes, root, attrs).build_lod()
    w, h = 120, 88
    r = renderer(yoxel_mod, w, h)
    r.SetScene(scene)
    r.SetDetailCoef(detail)
    assert_same(r.render_outputs(), oracle_frame(oracle, scene.nodes, scene.root, scene.attrs,
                                                 w, h, lod_coef=r.lod_coef()))


def test_batch_and_tiles(oracle, yoxel_mod):
    import torch
    w, h = 120, 88
    batch, keep = yoxel_mod.Batch(), []
    for k, p in enumerate(POOLS):
        nodes, root, attrs = pool(*p, 11 + k)
        r = renderer(yoxel_mod, w, h)
        r.SetSceneArrays(nodes, root, attrs)
        out = {k: torch.zeros((h, w), dtype=torch.float32 if k == "hit_t" else torch.int32,
                              device="cuda")
               for k in ("rgba", "hit", "hit_t", "fetches", "shadow_fetches")}
        batch.add_svo(r, **out)
        keep.append((r, out, oracle_frame(oracle, nodes, root, attrs, w, h)))
    batch.render()
    torch.cuda.synchronize()
    for r, out, ref in keep:
        assert_same(out, ref)
        part = {k: torch.zeros_like(v) for k, v in out.items()}
        tx, ty = r.tile_count()
        for b, e in ((0, 37), (37, 100), (100, tx * ty)):
            r.render_tiles(b, e, **part)
        torch.cuda.synchronize()
        assert_same(part, ref)
