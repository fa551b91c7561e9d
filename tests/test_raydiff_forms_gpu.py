"""The differentiable raycast's two forms evaluate one loss: raycast_loss and
raycast_loss_grad (with voxel gradients and without) give the same loss and
number of valid pixels bit for bit, as does raycast_loss_grad_masked under a
mask of every pixel, so a line search over the first continues the second."""
import numpy as np
import pytest
import torch

import synth
from superscanner_gb300 import GPUVoxelGrid
from superscanner_gb300.raydiff import raycast_loss, raycast_loss_grad, raycast_loss_grad_masked

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,vl", [("f32", 0.008), ("f16", 0.005)])
@pytest.mark.parametrize("rows,cols", [(60, 80), (97, 131), (240, 320)])
def test_forward_loss_is_the_gradient_forms(rows, cols, storage, vl):
    f = 525.0 * cols / 640
    intr = (f, f, (cols - 1) / 2, (rows - 1) / 2)
    sc = synth.Scene(2, 1234)
    P = sc.trajectory(6, 42)
    depth, _ = sc.render(P, rows, cols, intr, noise=True, noise_seed=7, color=False)
    dev = [torch.from_numpy(d.view(np.int16)).cuda() for d in depth]
    g = GPUVoxelGrid(int(1e9), 4 * vl, vl, rows, cols, storage=storage, with_color=False, hash_buckets=1 << 16)
    g.setIntrinsic(*intr)
    for k in range(5):
        g.integrate(None, dev[k], P[k].astype(np.float32), withColor=False)
    every = torch.ones((rows, cols), dtype=torch.uint8, device="cuda")
    voxels = torch.zeros((1 << 16, 512), device="cuda")
    for k in range(5):
        for lam in (0.0, 1.0):
            loss, valid = raycast_loss(g, P[k + 1], dev[k], lambda_n=lam)
            assert valid > 0.3 * rows * cols
            for form in (raycast_loss_grad(g, P[k + 1], dev[k], lambda_n=lam),
                         raycast_loss_grad(g, P[k + 1], dev[k], lambda_n=lam, grad_voxels=voxels),
                         raycast_loss_grad_masked(g, P[k + 1], dev[k], every, lambda_n=lam)):
                assert (form[0], form[2]) == (loss, valid)
    g.close()
