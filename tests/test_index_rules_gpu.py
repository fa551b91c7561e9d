"""The kernels' index rules on the device, against the reference's in
IEEE single precision, exactly: block and voxel of a point (voxel_of, block_of,
voxel_in_block), a projected voxel's pixel (project_axis_pair), a kokkosICP
window's centre (icp_center). Points next to every boundary, negative ones, past
2^22 voxels or pixels, infinities and NaN."""
import ctypes as C

import numpy as np
import pytest
import torch

from test_device_arith import _points

pytestmark = pytest.mark.gpu

F = np.float32
ODD = F([np.inf, -np.inf, np.nan, 0.0, -0.0, 1e-30, -1e-30, 1e-40, 3e9, -3e9, 1e30, 3e38, -3e38])


def _int(q):
    """(int) of a float as the device casts it: towards zero, clamped to the range, 0 for NaN."""
    q = np.nan_to_num(q.astype(np.float64), nan=0.0, posinf=1e300, neginf=-1e300)
    return np.clip(np.trunc(q), -2.0 ** 31, 2.0 ** 31 - 1).astype(np.int64).astype(np.int32)


def _rule(a, length):
    """getIndeces (GPUVoxelGrid.h:131-221): a >= 0 ? (int)(a / length) : (int)(a / length - 1)."""
    q = a / F(length)
    return np.where(a >= 0, _int(q), _int(q - F(1)))


def _ptr(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("length", [0.004, 0.0061, 0.02, 1.0 / 128])
def test_block_and_voxel_of_a_point(length):
    from superscanner_gb300._native import lib
    rng = np.random.default_rng(3)
    p = _points(F(length), rng)
    far = (2.0 ** rng.uniform(18, 32, 20000) * rng.choice([-1, 1], 20000) * length).astype(F)
    p = np.concatenate([p, far, np.nextafter(far, F(0)), np.tile(ODD, 50)])
    p = np.stack([p, rng.permutation(p), rng.permutation(p)], -1)
    dev = torch.from_numpy(p).cuda()
    out = torch.empty((len(p), 2, 4), dtype=torch.int32, device="cuda")
    assert lib.ss_test_voxel_index(_ptr(dev), len(p), float(length), _ptr(out), None) == 0
    torch.cuda.synchronize()
    with np.errstate(all="ignore"):
        vl = F(length)
        vbl = F(8) * vl
        b = _rule(p, vbl)
        v = _rule(p - vbl * b.astype(F), vl)
        # next to a block's face the rules can give an axis 8 or -1, and a place next to the block; further out: the nearest
        place = (v.astype(np.uint32) @ np.uint32([1, 8, 64])).view(np.int32)
        near = np.clip(v, 0, 7) @ np.int32([1, 8, 64])
        want = np.concatenate([b, np.where((place >= -512) & (place < 1024), place, near)[:, None]], -1)
    assert ((place < 0) | (place >= 512)).sum() > 1000
    got = out.cpu().numpy()
    assert np.array_equal(got[:, 1], want)
    assert np.array_equal(got[:, 0], want)


def _coordinates(rng, f, c, n):
    """(p, z) whose p f / z + c spread over and around an image of n pixels, a third of them next to a pixel's edge."""
    z = (rng.uniform(0.05, 12.0, 400_000) * rng.choice([1, 1, 1, -1], 400_000)).astype(F)
    t = rng.uniform(-1.5 * n, 2.5 * n, len(z))
    t[::3] = np.round(t[::3]) + rng.uniform(-2e-3, 2e-3, len(t[::3]))
    t[1::50] = 2.0 ** rng.uniform(18, 34, len(t[1::50])) * rng.choice([-1, 1], len(t[1::50]))
    p = ((t - c) * z.astype(np.float64) / f).astype(F)
    a, b = np.meshgrid(ODD, F([np.inf, -np.inf, np.nan, 0.0, -0.0, 1e-40, -1e-40, 1e-30, 1.0, -2.0, 1e30]))
    return np.concatenate([p, a.ravel(), a.ravel()[:1]]), np.concatenate([z, b.ravel(), b.ravel()[:1]])


@pytest.mark.parametrize("f,c,n", [(525.0, 319.5, 640), (131.25, 60.5, 120), (2100.0, 1279.5, 4096), (60.0, -3.0, 64),
                                   (-525.0, 239.5, 480)])
def test_pixel_of_a_projected_voxel(f, c, n):
    from superscanner_gb300._native import lib
    p, z = _coordinates(np.random.default_rng(4), f, c, n)
    p, z = p[:len(p) // 2 * 2], z[:len(p) // 2 * 2]
    dp, dz = torch.from_numpy(p).cuda(), torch.from_numpy(z).cuda()
    out = torch.empty(len(p), dtype=torch.int32, device="cuda")
    assert lib.ss_test_project(_ptr(dp), _ptr(dz), len(p), f, c, n, _ptr(out), None) == 0
    torch.cuda.synchronize()
    with np.errstate(all="ignore"):
        want = _int((p * F(f)) / z + F(c))
    got = out.cpu().numpy()
    inside = (want >= 0) & (want < n)
    assert inside.sum() > 50_000
    assert np.array_equal(got[inside], want[inside])
    assert not ((got >= 0) & (got < n))[~inside].any()


@pytest.mark.parametrize("rows,cols,fx,fy", [(480, 640, 525.0, 525.0), (97, 131, 107.0, -109.0), (720, 1280, 1050.0, 1049.0)])
def test_centre_of_an_icp_window(rows, cols, fx, fy):
    from superscanner_gb300._native import lib
    cx, cy = (cols - 1) / 2, (rows - 1) / 2
    rng = np.random.default_rng(5)
    x, z = _coordinates(rng, fx, cx, cols)
    i = rng.uniform(-20, rows + 20, len(z))
    i[::4] = np.round(i[::4]) + rng.uniform(-1e-3, 1e-3, len(i[::4]))
    with np.errstate(all="ignore"):
        y = ((i - (rows - cy)) * z.astype(np.float64) / fy).astype(F)
    z[7::97] = 0
    p = np.stack([x, y, z], -1)
    dev = torch.from_numpy(p).cuda()
    out = torch.empty((len(p), 3), dtype=torch.int32, device="cuda")
    assert lib.ss_test_icp_center(_ptr(dev), len(p), rows, cols, fx, fy, cx, cy, _ptr(out), None) == 0
    torch.cuda.synchronize()
    with np.errstate(all="ignore"):
        # the identity's products and sums: a coordinate next to an infinite or NaN one is NaN
        o = F(0)
        q = [((x + y * o) + z * o) + o, ((x * o + y) + z * o) + o, ((x * o + y * o) + z) + o]
        ci = _int((q[1] * F(fy)) / q[2] + (F(rows) - F(cy)))
        cj = _int((q[0] * F(fx)) / q[2] + F(cx))
    search = (z != 0) & (ci > 5) & (ci < rows - 5) & (cj > 5) & (cj < cols - 5)
    assert search.sum() > 50_000
    got = out.cpu().numpy()
    assert np.array_equal(got[:, 0] != 0, search)
    assert np.array_equal(got[search, 1], ci[search]) and np.array_equal(got[search, 2], cj[search])
