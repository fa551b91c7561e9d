"""kokkosICP's correspondence searches tap by tap: every pixel's chosen target
pixel is the one of a full scan of its window with the kernels' roundings (the
first smallest distance in the reference's order, kokkosICP.cpp:79-113): two of
a distance's products fused into its sum in windows read from shared memory,
every product rounded in those read from global memory."""
import ctypes as C

import numpy as np
import pytest
import torch

import synth
from test_device_arith import _rn32_exact
from test_icp_gpu import _motion

pytestmark = pytest.mark.gpu

F = np.float32
GLOBAL = 1 << 30  # ss_test_icp_taps' mark of a tile read from global memory


def _fma(a, b, c):
    """fma(a, b, c) of float32 arrays: a b is exact in float64, its sum with c a TwoSum pair, rounded once."""
    p, c = a.astype(np.float64) * b.astype(np.float64), c.astype(np.float64)
    hi = p + c
    v = hi - p
    return _rn32_exact(hi, (p - (hi - v)) + (c - v))


def _full_scan(src, dst, normals, T, intr, kind, fused=True):
    """(tap, the searched pixels, a warp's number of pixels that 16 taps do not settle) by all 100 taps."""
    rows, cols = src.shape[:2]
    fx, fy, cx, cy = (F(v) for v in intr)
    ci0, cj0 = F(rows) - cy, cx
    x, y, z = (src[..., k] for k in range(3))
    p = [((x * T[k, 0] + y * T[k, 1]) + z * T[k, 2]) + T[k, 3] for k in range(3)]
    with np.errstate(all="ignore"):
        ri, rj = (p[1] * fy) / p[2] + ci0, (p[0] * fx) / p[2] + cj0
    lost = ~(np.isfinite(ri) & np.isfinite(rj))
    ci, cj = (np.clip(np.where(lost, 0, np.trunc(v)), -1e6, 1e6).astype(np.int64) for v in (ri, rj))
    inside = (z != 0) & (ci > 5) & (ci < rows - 5) & (cj > 5) & (cj < cols - 5)
    at = np.nonzero(inside)
    q = np.stack([v[at] for v in p], -1)
    k, l = np.divmod(np.arange(100), 10)
    ti, tj = ci[at][:, None] + k - 5, cj[at][:, None] + l - 5
    t = dst[ti, tj]
    d = t - q[:, None, :]
    n = d if kind == 0 else normals[ti, tj]
    if fused:
        dot = _fma(d[..., 2], n[..., 2], _fma(d[..., 0], n[..., 0], d[..., 1] * n[..., 1]))
    else:
        dot = (d[..., 0] * n[..., 0] + d[..., 1] * n[..., 1]) + d[..., 2] * n[..., 2]
    dist = np.sqrt(dot) if kind == 0 else np.abs(dot)
    ok = (t[..., 2] != 0) & ((kind == 0) | (n[..., 0] != 0))
    dist = np.where(ok & (dist < F(0.075)), dist, F(np.inf))
    first = dist.argmin(1)
    rng = np.arange(len(first))
    tap = np.full((rows, cols), -1, np.int64)
    tap[at] = np.where(np.isfinite(dist[rng, first]), ti[rng, first] * cols + tj[rng, first], -1)
    # pixels whose nearest of the inner 4 x 4 taps is no nearer than a ray two pixels off may pass
    z2, fm = q[:, 2].astype(np.float64) ** 2, max(abs(float(fx)), abs(float(fy)))
    inner = dist[:, (k >= 4) & (k <= 7) & (l >= 4) & (l <= 7)].min(1)
    more = np.zeros((rows, cols), bool)
    more[at] = inner.astype(np.float64) ** 2 >= 4 * z2 * z2 / (fm * fm * (q.astype(np.float64) ** 2).sum(-1))
    wide = np.zeros((rows, -(-cols // 32) * 32), bool)
    wide[:, :cols] = more
    return tap, inside, wide.reshape(rows, -1, 32).sum(-1)


def _taps(d1, d2, tx, kind, intr, iteration):
    from superscanner_gb300 import depth_to_pcd, normals_from_pcd
    from superscanner_gb300._native import f64x16, lib
    dev = [torch.from_numpy(d.view(np.int16)).cuda() for d in (d1, d2)]
    rows, cols = d1.shape
    taps = torch.full((rows, cols), -2, dtype=torch.int32, device="cuda")
    txy = (C.c_float * 12)()
    assert lib.ss_test_icp_taps(C.c_void_p(dev[0].data_ptr()), C.c_void_p(dev[1].data_ptr()), rows, cols, *intr,
                                f64x16(tx), f64x16(np.eye(4)), kind, iteration, C.c_void_p(taps.data_ptr()), txy,
                                C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    src, dst = (depth_to_pcd(d, *intr) for d in dev)
    scene = (src.cpu().numpy(), dst.cpu().numpy(), normals_from_pcd(dst).cpu().numpy(),
             np.array(txy[:], F).reshape(3, 4), intr, kind)
    want, inside, more = _full_scan(*scene)
    got = taps.cpu().numpy().astype(np.int64)
    far = (got >= 0) & ((got & GLOBAL) != 0)
    if far.any():
        want = np.where(far, _full_scan(*scene, fused=False)[0], want)
    return np.where(far, got & ~GLOBAL, got), want, inside, more, far


def _room(rows, cols, deg, metres):
    f = 525.0 * cols / 640
    intr = (f, f, (cols - 1) / 2, (rows - 1) / 2)
    sc = synth.Scene(2, 77)
    P = sc.trajectory(6, 5)[[0, 4]]
    d, _ = sc.render(P, rows, cols, intr, noise=True, noise_seed=3, color=False)
    return d[1], d[0], np.linalg.inv(P[0]) @ _motion(deg, metres, rows) @ P[1], intr


@pytest.mark.parametrize("iteration", [0, 1, 9])
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("rows,cols,deg,metres", [(40, 53, 0.3, 0.004), (97, 131, 1.0, 0.02), (241, 321, 0.1, 0.001)])
def test_taps_of_a_room(rows, cols, deg, metres, kind, iteration):
    d1, d2, tx, intr = _room(rows, cols, deg, metres)
    got, want, inside, more, far = _taps(d1, d2, tx, kind, intr, iteration)
    assert inside.sum() > 0.5 * rows * cols
    if kind == 0 and (rows, cols) == (97, 131) and iteration == 0:  # both ways of a warp's pixels that need more taps
        assert ((more >= 1) & (more <= 8)).any() and (more > 8).any()
    assert np.array_equal(got, want)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("off", [(0.5, 0.0), (0.5, 0.5), (0.25, -0.5)])
def test_taps_that_nearly_tie(off, kind):
    """A slanted wall seen a fraction of a pixel off: the distances of two or four taps of a window (point to point), or
    of all its taps (point to plane), differ by their roundings alone."""
    rows, cols = 120, 160
    intr = (131.3, 131.7, 79.6, 59.4)
    i, j = np.mgrid[0:rows, 0:cols]
    flat = np.full((rows, cols), 1500, np.uint16)
    d = flat if kind == 0 else (1000 + 4 * j + i).astype(np.uint16)
    tx = np.eye(4)
    tx[:2, 3] = off[0] * 1.5 / 131.3, off[1] * 1.5 / 131.7
    got, want, inside, more, far = _taps(d, d, tx, kind, intr, 0)
    assert inside.sum() > 0.5 * rows * cols and not far.any()
    assert np.array_equal(got, want)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("rows,cols", [(96, 128), (131, 187)])
def test_taps_of_tiles_read_from_global_memory(rows, cols, kind):
    """Patches of two depths, seen from so far aside that the near ones move 0.35 of the image and the far ones a tenth:
    the windows of a tile lie too far apart for its staged region. Taps nearly tie as in the test above."""
    f = 0.82 * cols
    intr = (f, f, (cols - 1) / 2, (rows - 1) / 2)
    i, j = np.mgrid[0:rows, 0:cols]
    near = ((i // 8 + j // 8) % 2) == 0
    d = np.where(near, 700, 2500) if kind == 0 else np.where(near, 700 + j, 2500 + 3 * j)
    d = d.astype(np.uint16)
    tx = np.eye(4)
    tx[:2, 3] = (np.floor(0.35 * cols) + 0.5) * 0.7 / f, 0.5 * 0.7 / f
    got, want, inside, more, far = _taps(d, d, tx, kind, intr, 0)
    assert far.sum() > 500
    assert np.array_equal(got, want)
