"""ss_raycast along a block's face: where the reference's index rules name a
voxel outside the block (here layer 8 of 8, for every point of the rays in the
plane z = -2 block edges), the nearest voxel of the block is read, as the oracle
reads it, and never another block's memory."""
import numpy as np
import pytest
import torch

import oracle
from test_index_rules_gpu import _rule
from superscanner_gb300 import GPUVoxelGrid

pytestmark = pytest.mark.gpu

F = np.float32


@pytest.mark.parametrize("storage", ["f32", "f16"])
def test_rays_in_the_plane_of_a_negative_block_face(storage):
    vl = 1.0 / 128
    edge = 8 * vl
    z = F(-2 * edge)
    assert _rule(z - F(edge) * F(_rule(np.array([z]), F(edge))[0]), F(vl)) == 8
    rows, cols = 48, 64
    intr = (64.0, 64.0, 32.0, 24.0)  # the middle row's rays stay at the camera's z exactly
    E = np.eye(4, dtype=np.float32)
    E[:3, :3] = np.roll(np.eye(3), 1, 0)  # the camera looks along x, its rows go along y
    E[:3, 3] = 0.3 * edge, 0.4 * edge, -2 * edge
    depth = np.full((rows, cols), 1000, np.uint16)
    depth[:, 40:] = 800
    g = GPUVoxelGrid(int(1e9), 4 * vl, vl, rows, cols, storage=storage, with_color=False, hash_buckets=1 << 12)
    g.setIntrinsic(*intr)
    o = oracle.OracleGrid(vl, 4 * vl, rows, cols, intr=intr)
    g.integrate(None, torch.from_numpy(depth.view(np.int16)).cuda(), E, withColor=False)
    o.integrate(depth, None, E, with_color=False)
    got = g.raycast(E, with_color=False)[0].cpu().numpy()
    g.sync()
    g.close()
    want, _ = o.raycast(E)
    assert want.any(-1).mean() > 0.9 and (want[24, :, 2] == z).sum() > 50
    if storage == "f32":
        assert np.array_equal(got, want)
    else:  # the stored distances are rounded to 11 bits of the truncation
        assert np.array_equal(got.any(-1), want.any(-1))
        assert np.abs(got - want).max() <= 2.0 ** -11 * 4 * vl * 2
