"""The FP64 Gaussian's error against extended precision: on random keys its
mean is that of a correctly rounded square root and a cosine reduced to an
eighth of a turn (7.5e-17 relative, computed on the CPU for 3e6 keys; 8.0e-17 with a
root within an ulp and one polynomial over half a turn), and at the angles
where the reduction changes, the cosine's zeros among them, it stays within
the factors' bounds: half of 3.5e-16 (the logarithm under the root), 2^-53
(root), 2.3e-16 (cosine) and 2^-53 (product) (needs a GPU)."""
import ctypes as C

import numpy as np
import pytest

import legendre_b200 as L

pytestmark = pytest.mark.gpu

if np.finfo(np.longdouble).eps > 2.0 ** -63:
    pytest.skip("needs 80-bit long doubles", allow_module_level=True)

U64 = (1 << 64) - 1


def _mix(z):
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _unmix(z):  # the key that _mix maps to z
    def unshift(v, s):
        r = v
        for _ in range(64 // s + 1):
            r = v ^ (r >> s)
        return r

    z = unshift(z, 31) * pow(0x94D049BB133111EB, -1, 1 << 64) & U64
    z = unshift(z, 27) * pow(0xBF58476D1CE4E5B9, -1, 1 << 64) & U64
    return (unshift(z, 30) - 0x9E3779B97F4A7C15) & U64


def _error(sched, keys):
    keys = np.ascontiguousarray(keys, np.uint64)
    got = np.empty(keys.size)
    L._native.check(L._native.lib.lg_standard_normal(sched.handle, keys.ctypes.data_as(C.POINTER(C.c_uint64)),
                                                     keys.size, got.ctypes.data_as(C.POINTER(C.c_double))),
                    sched.handle)
    a = _mix(keys)
    b = _mix(a ^ np.uint64(0xD1B54A32D192ED03))
    u, v = (((z >> np.uint64(11)) + np.uint64(1)).astype(np.float64) * 2.0 ** -53 for z in (a, b))
    x = 6.283185307179586476925286766559 * v  # rounded to a double, as the reference does
    exact = np.sqrt(-2 * np.log(u.astype(np.longdouble))) * np.cos(x.astype(np.longdouble))
    return np.abs((got - exact) / exact).astype(np.float64)


def test_mean_error(sched):
    with np.errstate(over="ignore"):
        e = _error(sched, np.random.default_rng(3).integers(0, 1 << 63, 1 << 20, np.uint64) * np.uint64(2))
    assert e.mean() <= 7.6e-17
    assert e.max() <= 6.3e-16


def test_where_the_angle_changes_quadrant(sched):
    keys = []
    for eighth in range(8):
        for k in range(-40, 41):
            b = ((eighth << 61) + (k << 11)) & U64
            keys.append(_unmix(_unmix(b) ^ 0xD1B54A32D192ED03))
    with np.errstate(over="ignore"):
        e = _error(sched, keys)
    assert e.max() <= 6.3e-16
