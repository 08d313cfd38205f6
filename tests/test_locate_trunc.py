"""The fast voxel-location rule with the position truncated to FP32 by integer
operations (float_trunc and locate in physicore_gb300/csrc/cells_device.cuh), restated
with numpy: the truncation is exact towards zero over FP32's normal range, and
whenever the estimate decides, it agrees with the reference's FP64 expression
(mesh.cpp:37-61).  Positions as in test_locate_rule.py: every voxel boundary of several
meshes with offsets of 0..64 ulps, uniform, out of range, tiny and not finite."""
import numpy as np

from test_locate_rule import TOL_ABS, TOL_REL, adversarial_positions, reference


def float_trunc(p):
    """(valid, value) as the kernel evaluates it."""
    bits = p.astype(np.float64).view(np.uint64)
    hi, lo = (bits >> np.uint64(32)).astype(np.uint32), bits.astype(np.uint32)
    mag = hi & np.uint32(0x7fffffff)
    m = ((mag - np.uint32(896 << 20)) << np.uint32(3)) | (lo >> np.uint32(29))
    m = np.where(mag < np.uint32(897 << 20), np.uint32(0), m)
    f = ((hi & np.uint32(0x80000000)) | m).astype(np.uint32).view(np.float32)
    return mag < np.uint32(1151 << 20), f


def test_truncation():
    rng = np.random.default_rng(1)
    p = np.concatenate([rng.uniform(-1e6, 1e6, 100_000), np.ldexp(rng.uniform(1, 2, 10_000), rng.integers(-126, 127, 10_000)),
                        [0.0, -0.0, 1e-40, -1e-300, 2.0 ** -126, 16777217.0, 1.0 - 2.0 ** -53]])
    valid, f = float_trunc(p)
    assert valid.all()
    with np.errstate(over="ignore"):
        want = p.astype(np.float32)
    over = np.abs(want.astype(np.float64)) > np.abs(p)
    want = np.where(over, np.nextafter(want, np.float32(0)), want)
    want = np.where(np.abs(p) < 2.0 ** -126, np.float32(0), want)
    assert np.array_equal(f, want)
    assert not float_trunc(np.array([np.nan, np.inf, -np.inf, 1e39, 2.0 ** 128]))[0].any()


def test_truncated_rule_agrees_with_fp64_division():
    rng = np.random.default_rng(5)
    f32 = np.float32
    for bbmin, voxel, n in [(0, 20, 320), (0, 20, 200), (-100, 25, 37), (37, 7, 1000), (-2000, 10, 400), (5, 1, 4096),
                            (0, 3, 1), (-16777216, 16, 100_000)]:
        p = adversarial_positions(bbmin, voxel, n, rng)
        valid, pf = float_trunc(p)
        with np.errstate(invalid="ignore", over="ignore"):
            rf = f32(1.0 / voxel)
            qf = (pf - f32(bbmin)) * rf
            fl = np.floor(qf)
            tol = (np.abs(qf) + np.abs(pf) * rf) * TOL_REL + TOL_ABS
            decided = valid & ((qf - fl) > tol) & ((fl + f32(1.0)) - qf > tol)
        inside = (fl >= 0) & (fl < f32(n))
        ref_inside, ref_idx = reference(p, bbmin, voxel, n)
        assert np.array_equal(inside[decided], ref_inside[decided]), (bbmin, voxel, n)
        both = decided & ref_inside
        assert np.array_equal(fl.astype(np.float64)[both], ref_idx[both]), (bbmin, voxel, n)
        if abs(bbmin) < 1e6:  # with |p| / voxel near 2^20 the error bound reaches 1/2: nothing is decided
            assert decided[-200_007:-7].mean() > 0.99, (bbmin, voxel, n)
