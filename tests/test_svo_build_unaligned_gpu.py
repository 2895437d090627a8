"""GPU SVO build from grids that do not start on a 16-byte boundary (views into
larger arrays) against the CPU oracle of the build."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# depth 7 (128 voxels a row) is the first whose rows are read 16 bytes at a time
@pytest.mark.parametrize("off", [1, 2, 3, 4])
@pytest.mark.parametrize("depth", [6, 7])
def test_unaligned_grid(yoxel_mod, oracle, depth, off):
    import torch
    G = 1 << depth
    rng = np.random.default_rng(depth + off)
    d = (rng.standard_normal((G, G, G)) - 2.0).astype(np.float32)
    rgb = rng.integers(0, 256, (G, G, G, 3), dtype=np.uint8)
    bd = torch.zeros(d.size + 4, device="cuda")
    bc = torch.zeros(rgb.size + 4, dtype=torch.uint8, device="cuda")
    td = bd[off:off + d.size].view(d.shape)
    tc = bc[off:off + rgb.size].view(rgb.shape)
    td.copy_(torch.from_numpy(d))
    tc.copy_(torch.from_numpy(rgb))
    nodes, attrs, root = oracle.svo_build_dense(d, depth, 0.0, rgb)
    s = yoxel_mod.SVOScene.build_dense(td, depth, 0.0, tc)
    assert s.root == root and len(nodes) > 0
    assert np.array_equal(s.nodes_u32.reshape(-1, 10), nodes)
    assert np.array_equal(s.attrs_u8.reshape(-1, 8), attrs)
