"""The block set of an integrate call, and of a re-fusion, where the tiles'
bit boxes end: smooth tiles (all fit), white-noise depth (none fits), steps
(some fit), blocks small against the tile (more than 16 steps, more than four
of the second side), truncation of several blocks, odd image sizes and tile
heights. Exactly the oracle's set of blocks, weights and keys."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _depth(kind, rows, cols, seed):
    g = np.random.default_rng(seed)
    i, j = np.mgrid[0:rows, 0:cols]
    if kind == "ramp":
        d = 900 + 3.0 * j + 5.0 * i
    elif kind == "noise":
        d = g.uniform(250, 6000, (rows, cols))
    elif kind == "far":
        d = 5200 + 2.0 * j - 1.5 * i + g.normal(0, 20, (rows, cols))
    else:  # steps with holes
        d = 800 + 700 * ((j // 19 + i // 7) % 3) + g.normal(0, 3, (rows, cols))
        d[g.random((rows, cols)) < 0.2] = 0
    return d.astype(np.uint16)


def _pose(seed):
    g = np.random.default_rng(seed)
    q, _ = np.linalg.qr(g.normal(size=(3, 3)))
    T = np.eye(4, dtype=np.float32)
    T[:3, :3] = q * np.sign(np.linalg.det(q))
    T[:3, 3] = g.uniform(-1.5, 1.5, 3)
    return T


CASES = [("ramp", 48, 64, 0.004, 4), ("noise", 33, 37, 0.01, 4), ("far", 41, 97, 0.002, 4), ("steps", 40, 70, 0.005, 4),
         ("ramp", 25, 31, 0.01, 27), ("far", 8, 160, 0.004, 12), ("steps", 5, 3, 0.02, 2)]


def _grid(rows, cols, vl, trunc, intr, storage="f32"):
    from superscanner_gb300 import GPUVoxelGrid
    g = GPUVoxelGrid(int(1e8), trunc, vl, rows, cols, storage=storage, with_color=False, hash_buckets=1 << 18)
    g.setIntrinsic(*intr)
    return g


def _same(a, b):
    for k in ("keys", "coords", "w"):
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("tile_rows", [1, 4, 8])
@pytest.mark.parametrize("kind,rows,cols,vl,factor", CASES)
def test_blocks_of_a_frame(kind, rows, cols, vl, factor, tile_rows):
    intr = (70.0, 70.0, (cols - 1) / 2, (rows - 1) / 2)
    g = _grid(rows, cols, vl, factor * vl, intr)
    g.set_launch_config(collect_rows=tile_rows)
    o = oracle.OracleGrid(vl, factor * vl, rows, cols, intr=intr)
    for k in range(2):
        d, E = _depth(kind, rows, cols, k), _pose(10 * rows + k)
        g.integrate(None, torch.from_numpy(d.view(np.int16)).cuda(), E, False)
        o.integrate(d, None, E, with_color=False)
    g.sync()
    _same(g.export_blocks(with_color=False), o.export())


@pytest.mark.parametrize("kind,rows,cols,vl,factor", CASES)
def test_blocks_of_a_refusion(kind, rows, cols, vl, factor):
    intr = (70.0, 70.0, (cols - 1) / 2, (rows - 1) / 2)
    depths = [torch.from_numpy(_depth(kind, rows, cols, k).view(np.int16)).cuda() for k in range(3)]
    old, new = [_pose(5 + k) for k in range(3)], []
    for T in old:
        N = T.copy()
        N[:3, 3] += 0.02
        new.append(N)
    a, b = (_grid(rows, cols, vl, factor * vl, intr, "f16") for _ in range(2))
    for g in (a, b):
        for d, T in zip(depths, old):
            g.integrate_fast(d, T)
    a.refuse_batch(depths, old, new)
    for d, To, Tn in zip(depths, old, new):
        b.integrate_fast(d, To, deint=True)
        b.integrate_fast(d, Tn)
    a.sync(), b.sync()
    x, y = a.export_blocks(with_color=False), b.export_blocks(with_color=False)
    _same(x, y)
    assert np.array_equal(x["sdf"], y["sdf"])
