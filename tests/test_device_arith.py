"""CPU proofs of the kernels' exact-arithmetic shortcuts: a rewritten float
expression that must give the reference expression's IEEE single-precision
result for every input it can receive."""
import numpy as np


def _rn32_exact(hi, lo):
    """Round the exact value hi + lo (float64 pair, |lo| <= ulp(hi) / 2) to
    float32, ties to even."""
    r = hi.astype(np.float32)
    # hi on a float32 midpoint: the sign of lo decides, ties (lo == 0) to even
    up = np.nextafter(r, np.float32(np.inf))
    dn = np.nextafter(r, np.float32(-np.inf))
    mid_up = (r.astype(np.float64) + up.astype(np.float64)) / 2
    mid_dn = (r.astype(np.float64) + dn.astype(np.float64)) / 2
    r = np.where((hi == mid_up) & (lo > 0), up, r)
    r = np.where((hi == mid_dn) & (lo < 0), dn, r)
    return r


def test_depth_quotient_is_the_ieee_division_for_every_u16():
    """depth_m (ss_internal.cuh): RN(d / 1000) for every u16 d (the reference's
    (float)depth / 1000, GPUVoxelGrid.h:306) as q0 = RN(d y), y = RN(1/1000),
    r = fma(-q0, 1000, d), q = fma(r, y, q0)."""
    d = np.arange(65536, dtype=np.float32)
    want = d / np.float32(1000.0)  # IEEE single-precision division
    y = np.float32(1.0e-3)
    assert y == np.float32(1.0) / np.float32(1000.0)
    d64, y64 = d.astype(np.float64), np.float64(y)
    q0 = (d64 * y64).astype(np.float32)  # d y is exact in float64: one rounding
    rem = d64 - q0.astype(np.float64) * 1000.0  # exact in float64 (34-bit product, cancellation)
    r = rem.astype(np.float32)
    assert np.array_equal(r.astype(np.float64), rem)  # the fma's remainder is exact
    p = r.astype(np.float64) * y64  # exact (48-bit product)
    q0d = q0.astype(np.float64)
    hi = q0d + p
    bb = hi - q0d
    lo = (q0d - (hi - bb)) + (p - bb)  # TwoSum: hi + lo == q0 + p exactly
    got = _rn32_exact(hi, lo)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


# ------------------------------------------------ the voxel index shortcuts

F = np.float32


def _fma32(a, b, c):
    """fma(a, b, c) of float32 values to within the double rounding of a float64 sum (the margins tested below
    are compared against quantities that far larger steps separate)."""
    return (a.astype(np.float64) * np.float64(b) + np.float64(c)).astype(F)


def _idx_rule(a, length):
    q = a / F(length)
    return np.where(a >= 0, np.trunc(q), np.trunc(q - F(1))).astype(np.int64)


def _round_parts(a, rlen):
    """(floor of q, |q - rint(q)|, |q|) with q = RN(a rlen), as the kernels take them from 1.5 2^23 added and taken off."""
    q = a * F(rlen)
    t = q + F(12582912.0)
    d = q - (t - F(12582912.0))
    return (t.view(np.int32) - np.int32(0x4B400000) + (d.view(np.int32) >> 31)).astype(np.int64), np.abs(d), np.abs(q)


def _points(length, rng):
    """Coordinates over the packable range, most within a room, many within a few ulp of a voxel boundary."""
    lim = 8191 * 8 * float(length)
    u = np.concatenate([rng.uniform(-4, 4, 200_000), rng.uniform(-lim, lim, 100_000)]).astype(F)
    k = np.concatenate([rng.integers(-1200, 1200, 150_000), rng.integers(-65000, 65000, 50_000)])
    near = (k.astype(np.float64) * float(F(length))).astype(F)
    for _ in range(3):
        near = np.concatenate([near, np.nextafter(near[-len(k):], F(np.inf)), np.nextafter(near[:len(k)], F(-np.inf))])
    j = (k.astype(np.float64) * float(F(length)) * (1 + rng.uniform(-1e-5, 1e-5, len(k)))).astype(F)
    return np.concatenate([u, near, j, F([0.0, -0.0, 1e-30, -1e-30])])


def test_index_shortcuts_give_the_reference_rules():
    """idx_fast (ss_internal.cuh), idx_rule_fast and voxel_fast (ss_raycast.cu): where their tests are decisive, the block by
    idx_rule and the voxel by idx_rule of p - vbl block are those of the shortcut; and they are decisive for all but a
    few points of a room."""
    rng = np.random.default_rng(12)
    for length in (0.004, 0.005, 0.0061, 0.01, 0.02, 1.0 / 128):
        vl = F(length)
        vbl = F(8) * vl
        rvl, rvbl = F(1) / vl, F(1) / vbl
        p = _points(vl, rng)
        block = _idx_rule(p, vbl)
        b, d, q = _round_parts(p, rvbl)
        ok = d > _fma32(q, F(3.0e-7), F(3.0e-7))
        assert np.array_equal(b[ok], block[ok])
        w = p - vbl * block.astype(F)
        voxel = _idx_rule(w, vl)
        v, d, q = _round_parts(p, rvl)
        ok = d > _fma32(q, F(8.0e-7), F(1.6e-5))
        assert np.array_equal(v[ok] >> 3, block[ok]) and np.array_equal(v[ok] & 7, voxel[ok])
        assert ok[:200_000].mean() > 0.99
        bad = F([np.inf, -np.inf, np.nan, 3e9, -3e9])  # never decisive
        with np.errstate(invalid="ignore", over="ignore"):
            for r, m, c in ((rvbl, 3.0e-7, 3.0e-7), (rvl, 8.0e-7, 1.6e-5)):
                _, d, q = _round_parts(bad, r)
                assert not (d > _fma32(q, F(m), F(c))).any()


def test_projected_pixel_shortcut_gives_the_reference_cast():
    """project_axis_pair (ss_fuse.cuh): wherever its test is decisive, for any reciprocal within 1 ulp of 1 / z, its
    pixel is the truncated coordinate of the reference's IEEE quotient, or both lie outside the image; undecided only
    near pixel edges."""
    rng = np.random.default_rng(5)
    for f, c, n in ((525.0, 319.5, 640), (131.25, 60.5, 120), (2100.0, 1279.5, 4096), (60.0, -3.0, 64)):
        f, c = F(f), F(c)
        z = rng.uniform(0.05, 12.0, 400_000).astype(F) * rng.choice([1, 1, 1, -1], 400_000).astype(F)
        t = rng.uniform(-1.5 * n, 1.5 * n, 400_000)  # the pixel aimed at, a third of them next to an edge
        t[::3] = np.round(t[::3]) + rng.uniform(-2e-3, 2e-3, len(t[::3]))
        p = ((t - float(c)) * z.astype(np.float64) / float(f)).astype(F)
        pf = p * f
        want = np.trunc(pf / z + c).astype(np.int64)
        y = (1.0 / z.astype(np.float64)).astype(F)
        for rz in (y, np.nextafter(y, F(np.inf)), np.nextafter(y, F(-np.inf))):
            a = (pf.astype(np.float64) * rz.astype(np.float64) + float(c)).astype(F)
            fl = np.floor(a)
            decide = F(0.5) - F(4.0e-7) * (F(n + 2) + np.abs(c))
            sure = np.abs((a - fl) - F(0.5)) < decide
            got = fl.astype(np.int64) + (fl < 0)
            outside = ((got < 0) | (got >= n)) & ((want < 0) | (want >= n))
            assert (np.where(outside, want, got) == want)[sure].all()
            assert sure[1::3].mean() > 0.98
