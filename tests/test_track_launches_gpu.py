"""The launch-by-launch tracker over image sizes: CTAs and pixel groups that go
by a level's size."""
import numpy as np
import pytest
import torch

import synth
from superscanner_gb300 import GPUVoxelGrid
from superscanner_gb300.pipeline import Pipeline

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,levels", [
    (16, 16, 1), (24, 33, 2), (61, 97, 3), (120, 160, 3), (243, 323, 3), (480, 644, 2)])
def test_iteration_launches_of_any_size_match_the_persistent_tracker(rows, cols, levels):
    """The launch-by-launch tracker's CTAs and pixel groups go by a level's size; the persistent tracker's do not, and
    from the same model view both reach one pose, the solves differing by the roundings of the FP32 sums."""
    f = 0.8 * cols
    intr = (f, f, cols / 2 - 0.5, rows / 2 - 0.5)
    sc = synth.Scene(2, 77)
    P = sc.trajectory(4, 9)
    depth, _ = sc.render(P, rows, cols, intr, noise=True, noise_seed=3, color=False)
    poses = []
    for persistent in (False, True):
        g = GPUVoxelGrid(int(1e9), 0.04, 0.01, rows, cols, storage="f32", with_color=False, hash_buckets=1 << 16,
                         max_weight=255)
        g.setIntrinsic(*intr)
        pipe = Pipeline(g, use_graph=False, persistent_track=persistent, levels=levels)
        pipe.set_pose(P[0])
        for k in range(2):
            pipe.frame(torch.from_numpy(np.ascontiguousarray(depth[k].view(np.int16))).cuda(), track=k > 0)
        poses.append(pipe.pose())
    d = np.linalg.inv(poses[1]) @ poses[0]
    assert np.linalg.norm(d[:3, 3]) < 1e-5
    assert np.arccos(np.clip((np.trace(d[:3, :3]) - 1) / 2, -1, 1)) < 1e-5
