"""The fixed-point element arithmetic of the force and kinematics kernels
(lulesh_fixed*.cuh), the kernels' own functions compiled for the host, against
113-bit floating point.

Bounds, for an element with corner extent E and velocity extent dV. The scale
puts E in [2^60, 2^61), so a unit of a cross product of two differences (over
2^64) is at most 2^-56 E^2; an entry is off by at most a unit and a half (one
rounding down, two dropped lo*lo terms of a quarter each), and a double
rounds what it holds to 2^-53 of it.
  * volume derivatives (at most 3 E^2, sums of up to three entries):
    4.5 * 2^-56 + 3 * 2^-53 < 2^-50 of E^2;
  * 12 * volume: nine entries times at most 2 E, then 2.25 units of dropped
    terms, a unit over 2^128 being at most 2^-52 E^3: 27 * 2^-56 + 3 * 2^-52 +
    12 * 2^-53 < 2^-48 of E^3; taken elements hold at least 2^50 such units,
    so their relative error is below 4 * 2^-50 + 2^-53 < 2^-47;
  * squares of entries of at most 2 E^2: 2 * 2 * 1.5 * 3 * 2^-56 + 8 * 2^-53
    < 2^-49 of E^4, the edges' cross products alike (they are over 16);
  * sums against velocity differences: 2^-49 of 64 E^2 dV; the half-step
    determinant 2^-47 of 64 E^3;
  * base vectors are off by 2^-56 (three products of a derivative and a mode)
    at the strongest distortion 2^-52, so mode sums by 7 * 2^-52 + 8 * 2^-53 <
    2^-48 of dV, and forces, with |base vector| up to 13 there (the usual case:
    1), by 2^-44 of |s8| E^2 + |coef| dV; 2^-48 for a jitter of up to 5 % of E,
    where the base vectors stay below 2.
"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

CUBE = np.array([[0, 1, 1, 0, 0, 1, 1, 0], [0, 0, 1, 1, 0, 0, 1, 1], [0, 0, 0, 0, 1, 1, 1, 1]], float)


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    so = str(tmp_path_factory.mktemp("fixed") / "fixed_check.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off",
                    os.path.join(ROOT, "tests", "fixed_check.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)

    def forces(mode, pos, vel, scal):
        n = len(pos)
        taken, f, err = np.zeros(n, np.int32), np.zeros((n, 3, 8)), np.zeros((n, 4))
        L.check_forces(mode, n, _ptr(pos), _ptr(vel), _ptr(scal), _ptr(taken), _ptr(f), _ptr(err))
        return taken.astype(bool), f, err

    def kinematics(pos, vel, half_dt):
        n = len(pos)
        taken, err = np.zeros(n, np.int32), np.zeros((n, 13))
        L.check_kinematics(n, _ptr(pos), _ptr(vel), ctypes.c_double(half_dt), _ptr(taken), _ptr(err))
        return taken.astype(bool), err

    L.forces, L.kinematics = forces, kinematics
    return L


def _volume12(p):
    def d(a, b):
        return p[:, :, a] - p[:, :, b]
    t = ((d(3, 1) + d(7, 2), d(6, 3), d(2, 0)), (d(4, 3) + d(5, 7), d(6, 4), d(7, 0)),
         (d(1, 4) + d(2, 5), d(6, 1), d(5, 0)))
    return sum((u * np.cross(v, w)).sum(1) for u, v, w in t)


def _elements(seed, n, h, jitter, squash=1.0, shear=0.0):
    """n elements somewhere on a mesh of spacing h, on either side of the
    origin, jittered, squashed along z and sheared; velocities with an offset."""
    r = np.random.default_rng(seed)
    e = CUBE + jitter * r.uniform(-1, 1, (n, 3, 8))
    e[:, 2] *= squash
    e[:, 0] += shear * e[:, 1]
    pos = np.ascontiguousarray(h * (np.floor(r.uniform(-0.5 / h, 1 / h, (n, 3, 1))) + e))
    vel = np.ascontiguousarray(50 * (r.uniform(-1, 1, (n, 3, 1)) + 0.05 * r.uniform(-1, 1, (n, 3, 8))))
    scal = np.stack([1 / _volume12(pos), -0.03 * 80 * h * h * r.uniform(0, 1, n) * (r.random(n) < 0.8),
                     -r.uniform(0, 1e3, n) * (r.random(n) < 0.8) / 8], 1)
    return pos, vel, np.ascontiguousarray(scal)


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("h", [1.125 / 640, 1.125 / 150, 2.0 ** -7, 0.3, 40.0])
@pytest.mark.parametrize("jitter,squash,shear", [(0, 1, 0), (1e-9, 1, 0), (0.05, 1, 0), (0.2, 0.6, 0.4), (0.02, 0.2, 0)])
def test_forces(lib, mode, h, jitter, squash, shear):
    pos, vel, scal = _elements(3, 400, h, jitter, squash, shear)
    taken, force, err = lib.forces(mode, pos, vel, scal)
    assert taken.all() if squash == 1 else taken.any()
    err = err[taken]
    assert np.all(err[:, 1] <= 2.0 ** -50) and np.all(err[:, 2] <= 2.0 ** -49) and np.all(err[:, 3] <= 2.0 ** -48)
    assert np.all(err[:, 0] <= (2.0 ** -48 if jitter <= 0.05 and squash == 1 else 2.0 ** -44))


def test_forces_without_parts(lib):
    """No stress, no hourglass coefficient, neither, and a uniform motion: the
    missing part is exactly nothing."""
    pos, vel, scal = _elements(4, 50, 0.01, 0.05)
    scal[:, 1], scal[:, 2] = -1.0, -2.0
    both = lib.forces(0, pos, vel, scal)[1]
    for drop in ((1,), (2,), (1, 2)):
        s = scal.copy()
        s[:, list(drop)] = 0.0
        taken, f, err = lib.forces(0, pos, vel, s)
        assert taken.all() and np.all(err[:, 0] <= 2.0 ** -48)
        assert np.any(f != both)
    assert not lib.forces(0, pos, vel, np.stack([scal[:, 0], 0 * scal[:, 0], -0.0 * scal[:, 0]], 1).copy())[1].any()
    still = np.zeros_like(vel) + vel[:, :, :1]
    s = scal.copy()
    s[:, 1] = 0.0
    assert np.array_equal(lib.forces(0, pos, still, scal)[1], lib.forces(0, pos, still, s)[1])


@pytest.mark.parametrize("h", [1.125 / 640, 1.125 / 150, 2.0 ** -7, 0.3, 40.0])
@pytest.mark.parametrize("jitter,squash,shear", [(0, 1, 0), (1e-9, 1, 0), (0.05, 1, 0), (0.2, 0.6, 0.4), (0.02, 0.2, 0)])
def test_kinematics(lib, h, jitter, squash, shear):
    pos, vel, _ = _elements(5, 400, h, jitter, squash, shear)
    for half_dt in (0.0, h * 1e-6, h * 0.01):
        taken, err = lib.kinematics(pos, vel, half_dt)
        assert taken.all() if squash == 1 else taken.any()
        err = err[taken]
        assert np.all(err[:, 0] <= 2.0 ** -48) and np.all(err[:, 1:5] <= 2.0 ** -49)
        assert np.all(err[:, 5:9] <= 2.0 ** -49) and np.all(err[:, 9] <= 2.0 ** -47)
        assert np.all(err[:, 10] <= 2.0 ** -47) and np.all(err[:, 12] <= 2.0 ** -48)


@pytest.mark.parametrize("squash", [0.5, 0.25, 0.125, 0.06, 0.03, 0.015, 0.007])
def test_thin_elements_are_taken_with_full_accuracy_or_not_at_all(lib, squash):
    """Over extents through an octave, an element is either left to the FP64
    form or its volume is good to 2^-47 of itself."""
    some = 0
    for h in np.exp2(np.linspace(-7, -6, 9)):
        pos, vel, scal = _elements(6, 100, h, 0.02 * squash, squash, 0.3)
        taken, err = lib.kinematics(pos, vel, h * 1e-4)
        also = lib.forces(0, pos, vel, scal)[0]
        assert np.all(err[taken][:, 10] <= 2.0 ** -47)
        some += int(taken.sum()) + int(also.sum())
    assert some == 0 if squash < 0.01 else some > 0 if squash > 0.1 else True


def test_what_is_not_taken(lib):
    """Inverted, flat, tiny, huge and non-finite elements, wild scalars and
    velocities, a step that moves corners by more than the element."""
    pos, vel, scal = _elements(7, 12, 0.01, 0.02)
    bad = pos.copy()
    bad[0, 2] = bad[0, 2, 0]
    bad[1, 0] *= -1
    bad[2] *= 1e-4
    bad[3] *= 1e15
    bad[4, 1, 3] = np.nan
    bad[5, 0, 7] = np.inf
    bad[6, 0, 7] = -np.inf
    bad[7, 2, 2] = -np.nan
    vel_bad = vel.copy()
    vel_bad[8, 0, 0] = np.nan
    vel_bad[9, 1, 5] = -np.inf
    vel_bad[10, 2, 5] = 1e140
    taken, _ = lib.kinematics(bad, vel_bad, 1e-6)
    assert taken.tolist() == [False] * 11 + [True]
    taken, _, _ = lib.forces(0, bad, vel_bad, scal)
    assert taken.tolist() == [False] * 11 + [True]
    assert not lib.kinematics(pos, vel, 0.1)[0].any()  # corners move by half a volume's edge and more
    assert not lib.kinematics(pos, vel, np.nan)[0].any()
    for col, v in ((0, 0.0), (0, -1.0), (0, np.inf), (0, np.nan), (0, 1e-200), (1, np.nan), (1, np.inf), (1, 1e-200),
                   (2, np.nan), (2, -np.inf), (2, 1e200)):
        s = scal.copy()
        s[:, col] = v
        assert not lib.forces(0, pos, vel, s)[0].any(), (col, v)


def test_conversions(lib):
    """to_fixed modulo 2^64 and to_float, over signs, zeros, subnormals and
    shifts to both sides."""
    r = np.random.default_rng(8)
    x = np.concatenate([r.standard_normal(200), 1.125 * r.random(200), 2.0 ** r.integers(-60, 2, 200), -(2.0 ** r.integers(-60, 2, 200)),
                        [0.0, -0.0, 5e-324, -5e-324, 1.0, -1.0, np.nextafter(2, 0)]])
    bias = r.integers(8 - 1023 - 20, 8 - 1023 + 26, x.size).astype(np.int32)
    fixed, mant, expo = np.zeros(x.size, np.int64), np.zeros(x.size, np.int64), np.zeros(x.size, np.int32)
    lib.convert(x.size, _ptr(x), _ptr(bias), _ptr(fixed), _ptr(mant), _ptr(expo))
    for i in range(x.size):
        m, d = int(abs(x[i]) * 2.0 ** 60) if abs(x[i]) >= 2.0 ** -900 else 0, 60
        s = int(bias[i]) + 1075  # x 2^s, magnitude rounded down, then complemented when negative
        f = m << (s - d) if s >= d else m >> (d - s)
        num, den = float(abs(x[i])).as_integer_ratio()
        f = (num << s) // den if s >= 0 else num // (den << -s)
        f = -f - 1 if np.signbit(x[i]) else f
        assert (f - int(fixed[i])) % (1 << 64) == 0, (x[i], s)
        if abs(x[i]) >= 2.0 ** -1022:
            assert mant[i] * 2.0 ** int(expo[i]) == x[i] and 2 ** 60 <= abs(mant[i]) < 2 ** 61
        else:
            assert mant[i] == 0


def test_extents(lib):
    """The bound's exponent is at or just above that of max - min."""
    r = np.random.default_rng(9)
    v = np.concatenate([r.standard_normal((300, 8)), 100 + r.random((300, 8)), -100 - r.random((300, 8)),
                        2.0 ** r.integers(-40, 40, (300, 8)), np.zeros((1, 8)), -np.zeros((1, 8))])
    field = np.zeros(len(v), np.int32)
    lib.extents(len(v), _ptr(np.ascontiguousarray(v)), _ptr(field))
    for row, f in zip(v, field):
        ext = row.max() - row.min()
        assert ext < 2.0 ** (int(f) - 1022) or ext == 0
        assert 2.0 ** (int(f) - 1023) <= ext + 2.0 ** -18 * np.abs(row).max() + 1e-300
