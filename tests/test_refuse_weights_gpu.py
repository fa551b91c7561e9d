"""A batched re-fusion of a volume with weights that no fusion makes (an
imported volume's: fractions, negative, huge, infinite, NaN) gives the weights
and values of the sequential calls, bit for bit, NaN where they give NaN."""
import numpy as np
import pytest
import torch

import synth
from superscanner_gb300 import GPUVoxelGrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("max_weight", [0.0, 5.0])
def test_refusion_of_unusual_weights(max_weight, exact):
    rows, cols = 60, 80
    intr = (65.6, 65.6, 39.5, 29.5)
    sc = synth.Scene(2, 1234)
    P = sc.trajectory(4, 42)
    depth, _ = sc.render(P, rows, cols, intr, noise=True, noise_seed=7, color=False)
    dev = [torch.from_numpy(d.view(np.int16)).cuda() for d in depth]
    g = GPUVoxelGrid(int(1e9), 0.04, 0.01, rows, cols, storage="f32", with_color=False, hash_buckets=1 << 14,
                     max_weight=max_weight)
    g.setIntrinsic(*intr)
    for k in range(4):
        g.integrate(None, dev[k], P[k].astype(np.float32), withColor=False)
    start = g.export_blocks(with_color=False)
    w = start["w"].copy()
    pick = np.random.default_rng(9).random(w.shape)
    for k, v in enumerate((np.nan, np.inf, -np.inf, -1.0, 0.5, 3e38, 1e-40, -0.0)):
        w[(pick >= 0.02 * k) & (pick < 0.02 * (k + 1))] = v
    T_new = P.copy()
    T_new[:, 0, 3] += 0.02
    out = []
    for batched in (False, True):
        g.reset()
        g.import_blocks(start["coords"], start["sdf"], w)
        if batched:
            g.refuse_batch(dev, P, T_new, exact=exact)
        else:
            for k in range(4):
                if exact:
                    g.deIntegrate(None, dev[k], P[k].astype(np.float32), withColor=False)
                    g.integrate(None, dev[k], T_new[k].astype(np.float32), withColor=False)
                else:
                    g.integrate_fast(dev[k], P[k].astype(np.float32), deint=True)
                    g.integrate_fast(dev[k], T_new[k].astype(np.float32))
        g.sync()
        out.append(g.export_blocks(with_color=False))
    a, b = out
    g.close()
    assert np.isnan(a["w"]).sum() > 1000
    assert np.array_equal(a["keys"], b["keys"]) and np.array_equal(a["coords"], b["coords"])
    assert np.array_equal(a["w"], b["w"], equal_nan=True)
    assert np.array_equal(a["sdf"], b["sdf"], equal_nan=True)
