"""Forms of the raycasts' marches: which warp and lane marches a pixel, and how
many of its samples a turn tells, never shows in its result."""
import numpy as np
import pytest
import torch

import oracle
import synth
from superscanner_gb300 import GPUVoxelGrid
from superscanner_gb300.pipeline import raycast_maps
from superscanner_gb300.raydiff import raycast_loss

pytestmark = pytest.mark.gpu


def small_grid(rows, cols, storage):
    f = 0.8 * cols
    intr = (f, f, cols / 2 - 0.5, rows / 2 - 0.5)
    sc = synth.Scene(2, 31)
    P = sc.trajectory(3, 5)
    depth, _ = sc.render(P, rows, cols, intr, noise=True, noise_seed=3, color=False)
    g = GPUVoxelGrid(int(1e9), 0.04, 0.01, rows, cols, storage=storage, with_color=False, hash_buckets=1 << 16,
                     max_weight=255)
    g.setIntrinsic(*intr)
    for k in range(3):
        g.integrate_fast(torch.from_numpy(np.ascontiguousarray(depth[k].view(np.int16))).cuda(),
                         P[k].astype(np.float32))
    return g, P[2].astype(np.float32)


@pytest.mark.parametrize("rows,cols,launch_rows,storage", [
    (1, 1, 8, "f32"), (3, 7, 4, "f16"), (4, 8, 4, "f32"), (5, 33, 8, "f16"), (31, 65, 16, "f32"),
    (61, 97, 2, "f16"), (61, 97, 1, "f32"), (120, 160, 8, "f16"),
])
def test_maps_without_hint(rows, cols, launch_rows, storage):
    # a hint of zeros leaves every ray its whole range, in row segments
    g, pose = small_grid(rows, cols, storage)
    g.set_launch_config(raycast_rows=launch_rows)
    v, n = raycast_maps(g, pose)
    zeros = torch.zeros((rows, cols), dtype=torch.int16, device="cuda")
    v0, n0 = raycast_maps(g, pose, hint_depth=zeros, hint_margin=0.04)
    g.sync()
    assert torch.equal(v.view(torch.int32), v0.view(torch.int32))
    assert torch.equal(n.view(torch.int32), n0.view(torch.int32))
    if rows * cols > 1000:
        assert (v[..., 3] > 0).float().mean() > 0.5


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 7), (4, 16), (9, 33), (119, 161), (304, 256), (305, 256)])
def test_reference_raycast(rows, cols):
    # 304 x 256 is the largest image of half-full warps on 152 SMs; the bound is
    # the one of every raycast here: points bit for bit on 99.9 % of the pixels
    f = 0.8 * cols
    intr = (f, f, cols / 2 - 0.5, rows / 2 - 0.5)
    sc = synth.Scene(2, 31)
    P = sc.trajectory(2, 5).astype(np.float32)
    depth, rgb = sc.render(P, rows, cols, intr, noise=True, noise_seed=3, color=True)
    g = GPUVoxelGrid(int(1e9), 0.04, 0.01, rows, cols, hash_buckets=1 << 16)
    g.setIntrinsic(*intr)
    o = oracle.OracleGrid(0.01, 0.04, rows, cols, intr)
    for k in range(2):
        g.integrate(torch.from_numpy(np.ascontiguousarray(rgb[k])).cuda(),
                    torch.from_numpy(np.ascontiguousarray(depth[k].view(np.int16))).cuda(), P[k])
        o.integrate(depth[k], rgb[k], P[k])
    pcd, _ = g.raycast(P[1])
    got, want = pcd.cpu().numpy(), o.raycast(P[1])[0]
    assert np.all(got == want, axis=-1).mean() >= 0.999
    if rows * cols > 1000:
        assert (want[..., 2] != 0).mean() > 0.9


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("max_steps", [1, 2, 7, 18, 19, 20, 21, 33, 128])
def test_march_ahead(storage, max_steps):
    # the differentiable raycast's march tells several invalid samples a turn; it
    # ends after the same steps as the view's, which takes them one by one, and
    # gives a ray the hit of a longer march or none
    g, pose = small_grid(61, 97, storage)
    obs = torch.zeros((61, 97), dtype=torch.int16, device="cuda")
    full, depth = torch.zeros((61, 97), device="cuda"), torch.zeros((61, 97), device="cuda")
    raycast_loss(g, pose, obs, max_steps=400, depth_out=full)
    raycast_loss(g, pose, obs, max_steps=max_steps, depth_out=depth)
    t_min, t_max = float(np.float32(0.2)), float(np.float32(10.0))  # the grid's depth range
    v, _ = raycast_maps(g, pose, max_steps=max_steps, t_min=t_min, t_max=t_max)
    g.sync()
    hit = (v[..., 3] > 0) & (full > 0)
    assert torch.equal(depth, torch.where(hit, full, torch.zeros_like(full)))
    if max_steps == 128:
        assert hit.float().mean() > 0.5
