"""Marching cubes on the GPU where its work split ends: the smallest table
(one of the bucket groups that a warp takes) and larger ones, blocks with and
without neighbours, more triangles than a layer's list holds, and a buffer smaller
than the mesh. Against the FP64 oracle's triangles of the same volume."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

VL, TRUNC = 0.01, 0.04


def _volume(coords, field, buckets, storage, seen=lambda p: np.ones(len(p), bool)):
    """A grid holding field(points) (as sdf / truncation) in the given blocks."""
    from superscanner_gb300 import GPUVoxelGrid
    g = GPUVoxelGrid(int(1e8), TRUNC, VL, 48, 64, storage=storage, with_color=False, hash_buckets=buckets)
    g.setIntrinsic(60.0, 60.0, 31.5, 23.5)
    v = np.arange(512)
    local = np.stack([v & 7, (v >> 3) & 7, v >> 6], axis=1)
    pts = ((np.asarray(coords)[:, None] * 8 + local) + 0.5) * VL
    sdf = field(pts.reshape(-1, 3)).reshape(len(coords), 512).astype(np.float32)
    w = seen(pts.reshape(-1, 3)).reshape(len(coords), 512).astype(np.float32)
    g.import_blocks(np.asarray(coords, np.int32), sdf, w)
    g.sync()
    return g


def _sorted(t):
    t = np.asarray(t, np.float64).reshape(-1, 9)
    return t[np.lexsort(np.round(t / 1e-4).T[::-1])]


def _oracle(g):
    d = g.export_blocks(with_color=False)
    o = oracle.MethodGrid64(VL, TRUNC, g.resi, g.resj)
    o.import_blocks(d["coords"], d["sdf"], d["w"])
    return o.extract_mesh("cubes")


def _checker(p):  # a sign change on every edge: the most triangles a cell and a layer can have
    s = np.floor(p / VL).astype(int).sum(axis=1) & 1
    return np.where(s, 0.5, -0.25) * TRUNC


def _sphere(p):
    return np.clip(np.linalg.norm(p - 0.11, axis=1) - 0.07, -TRUNC, TRUNC)


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("buckets,coords,field", [
    (32, [(0, 0, 0)], _checker),
    (64, [(0, 0, 0), (1, 0, 0), (0, 1, 0), (1, 1, 1)], _checker),
    (1024, [(x, y, z) for x in range(-1, 3) for y in range(-1, 3) for z in range(-1, 3)], _sphere),
])
def test_cubes_match_the_oracle(storage, buckets, coords, field):
    from superscanner_gb300.mesh import extract_triangles
    g = _volume(coords, field, buckets, storage, seen=lambda p: (np.floor(p[:, 0] / VL) != 5) | (p[:, 1] > 0.03))
    got, want = extract_triangles(g).cpu().numpy(), _oracle(g)
    assert len(got) == len(want) > 0
    # vertices: a few float32 roundings of coordinates below 0.3 m (ulp 3e-8), as triangles matched by centroid
    from scipy.spatial import cKDTree
    c32, c64 = got.reshape(-1, 3, 3).mean(axis=1), np.asarray(want).reshape(-1, 3, 3).mean(axis=1)
    assert cKDTree(c64).query(c32)[0].max() < 1e-6 and cKDTree(c32).query(c64)[0].max() < 1e-6


def test_a_small_buffer_takes_its_share_and_no_more():
    from superscanner_gb300._native import check, lib
    from superscanner_gb300.mesh import extract_triangles
    g = _volume([(0, 0, 0), (1, 0, 0), (0, 1, 0)], _checker, 64, "f32")
    whole = {t.tobytes() for t in extract_triangles(g).cpu().numpy()}
    for cap in (1, 31, 32, 33, 100):
        out = torch.full((cap + 64, 3, 3), -7.0, device="cuda")
        n = C.c_int64()
        check(lib.ss_grid_extract_mesh_cubes(g.handle, cap, C.c_void_p(out.data_ptr()), C.byref(n), None), "mesh")
        h = out.cpu().numpy()
        assert n.value >= len(whole) and (h[cap:] == -7.0).all()
        assert all(t.tobytes() in whole for t in h[:cap])
