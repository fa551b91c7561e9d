"""kokkosICP's correspondence searches against the oracle where their shortcuts
end: odd image sizes (partial tiles, windows at the border), starts so far off
that few pixels find their nearest tap in the window's inner squares, and a flat
wall seen half a pixel off, where taps tie."""
import numpy as np
import pytest
import torch

import oracle
import synth

pytestmark = pytest.mark.gpu


def _motion(deg, metres, seed):
    g = np.random.default_rng(seed)
    ax = g.normal(size=3)
    ax /= np.linalg.norm(ax)
    a = np.radians(deg)
    K = np.array([[0, -ax[2], ax[1]], [ax[2], 0, -ax[0]], [-ax[1], ax[0], 0]])
    T = np.eye(4)
    T[:3, :3] += np.sin(a) * K + (1 - np.cos(a)) * K @ K
    v = g.normal(size=3)
    T[:3, 3] = v / np.linalg.norm(v) * metres
    return T


def _run(d1, d2, tx, ty, kind, intr):
    from superscanner_gb300 import kokkos_icp
    dev = [torch.from_numpy(d.view(np.int16)).cuda() for d in (d1, d2)]
    T, rmse = kokkos_icp(dev[0], dev[1], tx, ty, kind, intr)
    To, rmse_o, _ = oracle.kokkos_icp(d1, d2, tx, ty, kind, intr)
    # the bounds the ICP parity tests hold: 1e-4 rad, 0.1 mm
    dT = np.linalg.inv(To) @ T
    assert np.arccos(np.clip((np.trace(dT[:3, :3]) - 1) / 2, -1, 1)) <= 1e-4
    assert np.linalg.norm(dT[:3, 3]) <= 1e-4


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("rows,cols,deg,metres", [(40, 53, 0.3, 0.004), (97, 131, 1.0, 0.02), (120, 160, 3.0, 0.06),
                                                  (241, 321, 0.1, 0.001), (389, 517, 2.0, 0.04)])
def test_icp_search_matches_oracle(rows, cols, deg, metres, kind):
    f = 525.0 * cols / 640
    intr = (f, f, (cols - 1) / 2, (rows - 1) / 2)
    sc = synth.Scene(2, 77)
    P = sc.trajectory(6, 5)[[0, 4]]
    d, _ = sc.render(P, rows, cols, intr, noise=True, noise_seed=3, color=False)
    _run(d[1], d[0], _motion(deg, metres, rows) @ P[1], P[0], kind, intr)


@pytest.mark.parametrize("offset", [0.0, 0.5, 1.0])
def test_icp_ties_take_the_first_tap(offset):
    rows, cols = 96, 128
    intr = (128.0, 128.0, 64.0, 48.0)  # exact pixel quotients: neighbouring taps of a flat wall tie exactly
    d = np.full((rows, cols), 1024, np.uint16)
    d[30:50, 40:70] = 896  # a step fixes the motion along the wall
    tx = np.eye(4)
    tx[0, 3] = offset * 1.024 / 128
    tx[1, 3] = -offset * 1.024 / 128
    _run(d, d, tx, np.eye(4), 0, intr)
