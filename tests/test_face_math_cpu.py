"""CPU checks of the single-box kernels' face arithmetic (nmhd_b200/csrc/
mhd_math.cuh), compiled for the host (tests/native/libcellcheck.so): the HLLD
flux and the minbee reconstruction are bitwise the oracle's, which is pinned
to the reference's own hlld.inl and interpolate() (src/library/hlld.inl:7-284,
src/library/mhd_solver.inlrb:137-155).

The kernels compute the single-star state only for the side(s) the fan
region's formula reads (none in regions 0 and 5, the upwind side in 1 and 4,
both sides' transverse parts in 2 and 3) with the reference's operations;
these tests cover every region, Bx = 0 and both signs of Bx, with the exact
float bit patterns compared.

Tolerance: bitwise (every float of every output)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import adcheck
from oracle import oracle

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(HERE, "native", "libcellcheck.so")
GAMMA = np.float32(5.0 / 3.0)
_lib = None


def lib():
    global _lib
    if _lib is None:
        # make rebuilds the library when mhd_math.cuh changed
        subprocess.run(["make", "-s", "-C", os.path.join(HERE, "native")], check=True)
        L = ctypes.CDLL(LIB)
        P = ctypes.c_void_p
        L.cellh_hlld_many_f32.argtypes = [ctypes.c_float, P, P, P, ctypes.c_long]
        L.cellh_reconstruct_f32.argtypes = [P, P, ctypes.c_long]
        L.cellh_reconstruct_ranged_f32.argtypes = [P, P, P, ctypes.c_long]
        L.cellh_means_f32.argtypes = [P, P, P, P, ctypes.c_long]
        L.cellh_face_f32.argtypes = [ctypes.c_float, P, P, P, P, P, ctypes.c_long]
        L.cellh_hlld_ranged_f32.argtypes = [ctypes.c_float, P, P, P, P, P, ctypes.c_long]
        _lib = L
    return _lib


def riemann_inputs(rng, n):
    """(bx, lr) float32 inputs over all six fan regions: subsonic states,
    supersonic flows both ways, Bx = 0, strong and weak fields, equal states."""
    lr = np.empty((n, 14), np.float32)
    lr[:, 0:2] = rng.uniform(0.3, 2.0, (n, 2))
    lr[:, 2:8] = rng.normal(0.0, 1.0, (n, 6))
    sup = np.arange(n) % 7 == 0
    lr[sup, 2:4] += rng.choice([-4.0, 4.0], (sup.sum(), 1))
    lr[:, 8:10] = rng.uniform(0.2, 2.0, (n, 2))
    lr[:, 10:14] = rng.normal(0.0, 1.0, (n, 4)) * rng.choice([1e-3, 1.0, 3.0], (n, 1))
    eq = np.arange(n) % 11 == 0
    lr[eq, 1::2] = lr[eq, 0::2]
    bx = rng.normal(0.0, 1.0, n).astype(np.float32) * rng.choice([1e-2, 1.0, 4.0], n).astype(np.float32)
    bx[np.arange(n) % 5 == 0] = 0.0
    return bx, np.ascontiguousarray(lr)


def test_device_hlld_is_bitwise_the_oracle_in_all_regions():
    rng = np.random.default_rng(11)
    n = 6000
    bx, lr = riemann_inputs(rng, n)
    out = np.empty((n, 7), np.float32)
    lib().cellh_hlld_many_f32(GAMMA, bx.ctypes.data, lr.ctypes.data, out.ctypes.data, n)
    regions = np.zeros(6, int)
    for i in range(n):
        ref = oracle.hlld(GAMMA, bx[i], lr[i], np.float32)
        assert np.array_equal(out[i].view(np.uint32), ref.view(np.uint32)), (i, bx[i], lr[i], out[i], ref)
        regions[adcheck.hlld_region(float(GAMMA), bx[i], lr[i])] += 1
    assert (regions > 50).all(), regions


@pytest.mark.parametrize("gamma, scale", [(5.0 / 3.0, 1.0), (1.4, 1e-3), (1.001, 1e3), (2.0, 1e-9), (5.0 / 3.0, 1e5)])
def test_ranged_hlld_is_the_plain_one_where_it_takes_the_state(gamma, scale):
    """hlld_flux_ranged against hlld_flux_plain (the reference's operations,
    bitwise the oracle's above), bit for bit, on states whose pressure and
    energies are of order `scale`; and that ordinary states are taken, tiny
    numerators, vacuum, infinities and NaN are not."""
    rng = np.random.default_rng(5)
    n = 200000
    bx, lr = riemann_inputs(rng, n)
    bx *= np.float32(np.sqrt(scale))
    lr[:, 2:8] *= np.float32(np.sqrt(scale))
    lr[:, 10:14] *= np.float32(np.sqrt(scale))
    lr[:, 8:10] *= np.float32(scale)
    quiet = np.arange(n) % 17 == 0  # nearly equal sides: small differences everywhere
    lr[quiet, 1::2] = lr[quiet, 0::2] * (1 + rng.normal(0, 1e-7, (quiet.sum(), 7))).astype(np.float32)
    zero = np.arange(n) % 19 == 0   # no transverse field
    lr[zero, 10:14] = 0
    odd = np.arange(n) < 8          # states that must be left to the plain path
    lr[0, 0] = 0
    lr[1, 8] = -lr[1, 8]
    lr[2, 4] = np.nan
    lr[3, 12] = np.inf
    lr[4, 0] = np.nan
    lr[5, 2] = np.inf
    lr[6, 2:8], lr[6, 10:14], bx[6] = 0, 1e-30, 1e-15
    bx[7] = np.nan
    out, ref, ok = np.empty((n, 7), np.float32), np.empty((n, 7), np.float32), np.empty(n, np.int32)
    lib().cellh_hlld_ranged_f32(gamma, bx.ctypes.data, lr.ctypes.data, out.ctypes.data, ref.ctypes.data, ok.ctypes.data, n)
    took = ok != 0
    assert not took[odd].any()
    assert took.mean() > (0.99 if 1e-6 < scale < 1e4 else 0.5), took.mean()
    assert np.array_equal(out[took].view(np.uint32), ref[took].view(np.uint32))


def test_device_reconstruction_is_the_minbee_limiter():
    """reconstruct4 against the reference's interpolate() restated in numpy
    (float32 operations): L = x1 + minmod(x1-x0, x2-x1)/2, R = x2 - minmod(x2-x1,
    x3-x2)/2, minmod 0 for products <= 0, else the smaller magnitude (ties: the
    second argument)."""
    rng = np.random.default_rng(3)
    n = 20000
    x = rng.normal(0.0, 1.0, (n, 4)).astype(np.float32)
    x[::9, 2] = x[::9, 1]          # zero slopes
    x[::13, 3] = 2 * x[::13, 2] - x[::13, 1]  # equal slopes (ties)
    lr = np.empty((n, 2), np.float32)
    lib().cellh_reconstruct_f32(np.ascontiguousarray(x).ctypes.data, lr.ctypes.data, n)
    f = np.float32

    def minmod(a, b):
        return np.where(a * b <= f(0), f(0), np.where(np.abs(a) < np.abs(b), a, b)).astype(np.float32)

    d01, d12, d23 = x[:, 1] - x[:, 0], x[:, 2] - x[:, 1], x[:, 3] - x[:, 2]
    left = x[:, 1] + minmod(d01, d12) / f(2)
    right = x[:, 2] - minmod(d12, d23) / f(2)
    assert np.array_equal(lr[:, 0].view(np.uint32), left.view(np.uint32))
    assert np.array_equal(lr[:, 1].view(np.uint32), right.view(np.uint32))


@pytest.mark.parametrize("scale", [1.0, 1e-20, 1e-30, 1e-42])
def test_ranged_reconstruction_is_the_plain_one_where_it_takes_the_slopes(scale):
    """reconstruct4_with against reconstruct4 (equal values; the sign of a zero
    may differ), on slopes of order `scale` on a zero and on a non-zero mean:
    taken unless a non-zero slope is below 2^-73."""
    rng = np.random.default_rng(13)
    n = 40000
    x = (rng.normal(0.0, 1.0, (n, 4)) * scale).astype(np.float32)
    x[::3] += np.float32(rng.choice([0.25, -3.0]))
    x[::9, 2] = x[::9, 1]
    x[::13, 3] = 2 * x[::13, 2] - x[::13, 1]
    x = np.ascontiguousarray(x)
    lr, ref, ok = np.empty((n, 2), np.float32), np.empty((n, 2), np.float32), np.empty(n, np.int32)
    lib().cellh_reconstruct_ranged_f32(x.ctypes.data, lr.ctypes.data, ok.ctypes.data, n)
    lib().cellh_reconstruct_f32(x.ctypes.data, ref.ctypes.data, n)
    took = ok != 0
    assert np.array_equal(lr[took], ref[took])
    assert took[::3].all() or scale == 1.0
    assert took.mean() > 0.95 if scale > 1e-21 else not took[1::3].all()


def assert_face_takes_only_what_it_computes_alike(bx, x):
    n = len(bx)
    a, b, ok = np.empty((n, 7), np.float32), np.empty((n, 7), np.float32), np.empty(n, np.int32)
    lib().cellh_face_f32(5.0 / 3.0, bx.ctypes.data, x.ctypes.data, a.ctypes.data, b.ctypes.data, ok.ctypes.data, n)
    took = ok != 0
    assert np.array_equal(a[took], b[took], equal_nan=True)


def face_cells(rng, n):
    """Four cells a face: density, velocities (some supersonic), pressure, sums of B."""
    x = rng.normal(0.0, 1.0, (n, 4, 7))
    x[:, :, 0] = rng.uniform(0.5, 2.0, (n, 4))
    x[:, :, 4] = rng.uniform(0.1, 2.0, (n, 4))
    x[:, :, 1] += rng.choice([0.0, 6.0, -6.0], (n, 1))
    return rng.normal(0.0, 0.5, n).astype(np.float32), x.astype(np.float32)


@pytest.mark.parametrize("value", [np.nan, -np.nan, np.inf, -np.inf])
def test_ranged_face_leaves_cells_that_are_not_finite_to_the_plain_one(value):
    """One value of one of a face's four cells is not finite: its flux by the shared
    reciprocals is the plain one, NaN for NaN, or is not taken."""
    rng = np.random.default_rng(17)
    n = 56000
    bx, x = face_cells(rng, n)
    at = np.arange(n)
    x[at, at % 4, at // 4 % 7] = np.float32(value)
    assert_face_takes_only_what_it_computes_alike(bx, np.ascontiguousarray(x))


def test_ranged_means_with_slopes_at_the_limiters_underflow():
    """Sums of two values with differences of a few 2^-75: the products of the means'
    slopes underflow to 0 below 2^-75, and the plain limiter is then off."""
    rng = np.random.default_rng(19)
    n = 40000
    s = (rng.integers(-24, 25, (n, 4)) * 2.0 ** -75).astype(np.float32)
    a, b, ok = np.empty((n, 2), np.float32), np.empty((n, 2), np.float32), np.empty(n, np.int32)
    lib().cellh_means_f32(s.ctypes.data, a.ctypes.data, b.ctypes.data, ok.ctypes.data, ctypes.c_long(n))
    took = ok != 0
    assert 0.05 < took.mean() < 0.95
    assert np.array_equal(a[took], b[took])


@pytest.mark.parametrize("cell, likely", [
    ((1.0, 1.0, 0.0, 0.0, 0.0), True), ((1.0, 1.0, 1e-3, 0.0, 1e-9), True),
    ((1.0, 1.0, 0.5, 1e-20, -1e-13), True),  # one strong component
    ((1.0, 1.0, 1e-12, -1e-13, 0.0), False), ((1.0, 1.0, 0.0, 0.0, -1e-30), False),
    ((2.0 ** -46, 1.0, 0.1, 0.1, 0.1), False), ((1.0, 2.0 ** 30, 0.1, 0.1, 0.1), False), ((1.0, -1.0, 0.1, 0.1, 0.1), False),
    ((np.nan, 1.0, 0.1, 0.1, 0.1), False)])
def test_cells_whose_faces_are_unlikely_to_hold(cell, likely):
    f = lib().cellh_likely_in_range
    f.argtypes = [ctypes.c_float] * 5
    assert bool(f(*cell)) == likely
