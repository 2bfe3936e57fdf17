"""The WET smoothing's constant index offsets (dc_wet_smooth_offsets) against the reference's own float32
expression, evaluated voxel by voxel in NumPy: rotate the voxel into the head frame, step dr along the
direction, rotate back, (int)roundf((q + iso) / spacing) (IMPTClasses.cu:139-202, CudaClasses.cuh:112-116).
On an axis without the exact bit the offset must hold for every voxel, whether or not the compiler fuses the
rotations' multiply-adds."""
import ctypes as C

import numpy as np
import pytest

from dosecuda_b200 import _lib

F = np.float32


def _offsets(shape, spacing, origin, iso, gantry, couch):
    out = (C.c_int * (54 * 4))()
    _lib.raise_for(_lib.load().dc_wet_smooth_offsets(*shape, _lib.f3(spacing), _lib.f3(origin), _lib.f3(iso), gantry, couch,
                                                     1635.0, out))
    return np.array(out).reshape(54, 4)


def _mul_add(a, b, c, d, fused):
    """a*b + c*d in float32: each step rounded, or the second product fused into the sum."""
    if fused:
        return (a.astype(np.float64) * b + (c * d).astype(F).astype(np.float64)).astype(F)
    return ((a * b).astype(F) + (c * d).astype(F)).astype(F)


def _reference(ijk, spacing, origin, iso, gantry, couch, fused):
    iso_rel = (np.asarray(iso, F) - np.asarray(origin, F)).astype(F)
    sp = np.asarray(spacing, F)
    ga = F(F((gantry + 180.0) % 360.0) * F(np.pi) / F(180.0))
    ta = F(F(couch) * F(np.pi) / F(180.0))
    sga, cga, sta, cta = (F(f(float(a))) for a in (ga, ta) for f in (np.sin, np.cos))
    p = ((ijk.astype(F) * sp).astype(F) - iso_rel).astype(F)
    xt = _mul_add(p[:, 0], cta, p[:, 2], F(-sta), fused)
    zt = _mul_add(p[:, 0], sta, p[:, 2], cta, fused)
    xg = _mul_add(xt, cga, p[:, 1], sga, fused)
    yg = _mul_add(xt, F(-sga), p[:, 1], cga, fused)
    h = np.stack((-xg, zt, yg), 1)
    for d in range(6):
        ang = F(F(d) * F(np.pi)) / F(3.0)
        s, co = F(np.sin(float(ang))), F(np.cos(float(ang)))
        for dr in range(1, 10):
            hx = (h[:, 0] + F(dr) * co).astype(F)
            hy = (h[:, 1] + F(dr) * s).astype(F)
            x, y, z = -hx, h[:, 2], hy
            xg2 = _mul_add(x, cga, y, F(-sga), fused)
            yg2 = _mul_add(x, sga, y, cga, fused)
            q = np.stack((_mul_add(xg2, cta, z, sta, fused), yg2, _mul_add(xg2, F(-sta), z, cta, fused)), 1)
            v = ((q + iso_rel).astype(F) / sp).astype(F)
            yield (np.sign(v) * np.floor(np.abs(v).astype(np.float64) + 0.5)).astype(np.int64)


@pytest.mark.parametrize("spacing,gantry,couch", [
    ((2.0, 2.0, 2.0), 0.0, 0.0), ((1.0, 1.0, 1.0), 90.0, 0.0), ((2.5, 2.5, 2.5), 180.0, 0.0), ((1.5, 1.5, 2.0), 71.7, 0.0),
    ((2.0, 2.0, 2.5), 235.0, 30.0), ((3.0, 3.0, 3.0), 30.0, 10.0), ((0.9765625, 0.9765625, 3.0), 310.0, -45.0),
    ((1.2, 2.4, 0.7), 270.0, 0.0), ((4.0, 1.0, 2.0), 45.0, 90.0)])
def test_constant_offsets_are_the_reference_index(spacing, gantry, couch):
    shape = (150, 260, 256)
    rng = np.random.default_rng(int(gantry) + int(10 * spacing[0]))
    origin = np.array([-n * s / 2 for n, s in zip(shape[::-1], spacing)]) + rng.uniform(-40, 40, 3)
    iso = rng.uniform(-60, 60, 3)
    if gantry in (0.0, 90.0):  # isocentre on a voxel centre: every second sample sits on a half-integer
        iso = origin + np.array([120, 130, 70]) * np.asarray(spacing)
    ijk = np.stack([rng.integers(0, n, 4000) for n in shape[::-1]], 1)
    table = _offsets(shape, spacing, origin, iso, gantry, couch)
    free = 0
    for fused in (False, True):
        for e, index in enumerate(_reference(ijk, spacing, origin, iso, gantry, couch, fused)):
            for a in range(3):
                # marked axes: the constant offset or one beside it (the kernel's reach)
                assert np.abs(index[:, a] - ijk[:, a] - table[e, a]).max() <= 1
                if not table[e, 3] >> a & 1:
                    free += 1
                    assert np.array_equal(index[:, a], ijk[:, a] + table[e, a]), (e, a)
    assert free >= 0.75 * 2 * 54 * 3  # most samples need no per-voxel evaluation


def test_offsets_reject_null_and_survive_extreme_spacings():
    lib = _lib.load()
    assert lib.dc_wet_smooth_offsets(1, 1, 1, _lib.f3((1, 1, 1)), _lib.f3((0, 0, 0)), _lib.f3((0, 0, 0)), 0.0, 0.0, 1.0,
                                     None) == _lib.DC_ERR_VALUE
    t = _offsets((8, 8, 8), (1e-5, 1e-5, 1e-5), (0, 0, 0), (0, 0, 0), 33.0, 0.0)  # offsets beyond any table
    assert (t[:, 3] != 0).all()
    t = _offsets((8, 8, 8), (100.0, 100.0, 100.0), (0, 0, 0), (0, 0, 0), 33.0, 0.0)  # every sample in the voxel itself
    assert (t == 0).all()
