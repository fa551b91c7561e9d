"""ss_raycast where the reference's index rules name a place outside of a block:
the table's last block has an empty one behind it, so a ray that reads on there
sees an unobserved voxel and goes through."""
import numpy as np
import pytest

from test_index_rules_gpu import _rule
from superscanner_gb300 import GPUVoxelGrid

pytestmark = pytest.mark.gpu

F = np.float32


@pytest.mark.parametrize("with_color", [False, True])
@pytest.mark.parametrize("storage", ["f32", "f16"])
def test_a_read_behind_the_last_block_is_empty(storage, with_color):
    vl, rows, cols, buckets = 1.0 / 128, 48, 64, 32
    edge = 8 * vl
    z = F(-2 * edge)  # at a negative multiple of the edge the rules give block -3 and its layer 8 of 8
    assert _rule(np.array([z]), F(edge))[0] == -3 and _rule(z - F(edge) * F(-3), F(vl)) == 8
    sdf = np.zeros((1, 8, 8, 8), np.float32)  # [z, y, x]: a surface across x, seen from smaller x
    sdf[..., :4], sdf[..., 4:] = 2 * vl, -2 * vl
    for bx in range(400):  # a block that lands in the last bucket
        g = GPUVoxelGrid(int(1e9), 4 * vl, vl, rows, cols, storage=storage, with_color=with_color, hash_buckets=buckets)
        g.import_blocks([[bx, 0, -3]], sdf.reshape(1, 512), np.ones((1, 512), np.float32),
                        np.zeros((1, 3, 512), np.float32) if with_color else None)
        if g.export_buckets()[0] == buckets - 1:
            break
        g.close()
    else:
        pytest.fail("no block in the last bucket")
    g.setIntrinsic(640.0, 640.0, 32.0, 24.0)
    E = np.eye(4, dtype=np.float32)
    E[:3, :3] = np.roll(np.eye(3), 1, 0)  # looks along x, columns along y, rows along z: row 24 stays at z
    E[:3, 3] = bx * edge - 0.5, 0.5 * edge, z
    view = g.raycast(E, with_color=with_color)[0].cpu().numpy()
    g.sync()
    g.close()
    hit = view.any(-1)
    assert not hit[24:].any()  # row 24: the empty block behind the last; the rows above it: no block
    # below it the surface, where the reference's interpolation puts it: 2.5 voxels behind the centre of voxel 3
    assert hit[10:23, 32].all() and np.abs(view[10:23, 32, 0] - (bx * edge + 6 * vl)).max() < vl
