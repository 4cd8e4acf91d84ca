"""The kinematics' fixed-point sums (lulesh_fixed_kin.cuh) and the corner forces
(lulesh_fixed_force.cuh) beside the FP64 expressions they took the place of, both against 113-bit floating point: over a
group of elements the largest error, relative to the sum of the magnitudes of the
sum's products, may not be larger than that of the FP64 expressions by more than
2^-52 (a result rounded to a double, 2^-53 of the sum, and as much again for
cuts at 2^-56 and below). A bound over the element's box cannot see a direction,
or a velocity component, far below the others.
"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

CUBE = np.array([[0, 1, 1, 0, 0, 1, 1, 0], [0, 0, 1, 1, 0, 0, 1, 1], [0, 0, 0, 0, 1, 1, 1, 1]], float)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    so = str(tmp_path_factory.mktemp("sizes") / "sizes.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off",
                    os.path.join(ROOT, "tests", "fixed_sizes_check.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.fixture(scope="module")
def sums(lib):
    def run(pos, vel, half_dt, wide=False):
        n = len(pos)
        taken = np.zeros(n, np.int32)
        out = [np.zeros((n, 10)) for _ in range(4)]
        lib.check_sizes(int(wide), n, *(a.ctypes.data_as(ctypes.c_void_p) for a in (pos, vel)), ctypes.c_double(half_dt),
                        *(a.ctypes.data_as(ctypes.c_void_p) for a in (taken, *out)))
        return taken.astype(bool), *out  # want, errors of the fixed-point and the FP64 form, size
    return run


@pytest.fixture(scope="module")
def forces(lib):
    def run(pos, vel, scal, wide=False):
        n = len(pos)
        taken = np.zeros(n, np.int32)
        out = [np.zeros((n, 3)) for _ in range(3)]
        lib.check_force_sizes(int(wide), n, *(a.ctypes.data_as(ctypes.c_void_p) for a in (pos, vel, np.ascontiguousarray(scal), taken, *out)))
        return taken.astype(bool), *out  # errors of the fixed-point and the FP64 form, size
    return run


def _elements(seed, n, h, jitter, squash=1.0, axis=2, ratio=1.0):
    """n elements on a mesh of spacing h, jittered and squashed along an axis;
    velocities whose differences along x are 1/ratio those of y and z."""
    r = np.random.default_rng(seed)
    e = CUBE + jitter * r.uniform(-1, 1, (n, 3, 8))
    e[:, axis] *= squash
    pos = np.ascontiguousarray(h * (np.floor(r.uniform(0, 1 / h, (n, 3, 1))) + e))
    vel = r.uniform(-1, 1, (n, 3, 8))
    vel[:, 1:] *= ratio
    return pos, np.ascontiguousarray(vel)


def _no_further_off(fixed, fp64, size, which):
    for j in which:
        assert (fixed[:, j] / size[:, j]).max() <= (fp64[:, j] / size[:, j]).max() + 2.0 ** -52, j


@pytest.mark.parametrize("h", [1.125 / 150, 2.0 ** -7, 0.3])
@pytest.mark.parametrize("jitter", [0.0, 1e-6, 0.05])
@pytest.mark.parametrize("ratio", [1.0, 1e-3, 1e-6, 1e-9, 1e-10, 1e-12])
def test_velocity_sums_in_flow_along_one_axis(sums, h, jitter, ratio):
    pos, vel = _elements(1, 200, h, jitter, ratio=ratio)
    for half_dt in (0.0, 1e-3 * h):
        taken, _, fixed, fp64, size = sums(pos, vel, half_dt)
        assert taken.all()
        _no_further_off(fixed, fp64, size, range(5, 9))


@pytest.mark.parametrize("h", [1.125 / 30, 1.125 / 150, 2.0 ** -7])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("squash", [1.0, 0.5, 0.2, 0.09, 1 / 25, 1 / 32])
def test_sums_of_thin_elements(sums, h, axis, squash):
    pos, vel = _elements(2, 400, h, 0.02, squash, axis)
    taken, _, fixed, fp64, size = sums(pos, vel, 1e-4 * h)
    assert taken.all() if squash > 0.1 else taken.any()
    _no_further_off(fixed[taken], fp64[taken], size[taken], range(10))


@pytest.mark.parametrize("boost", [1.0, 1e3, 1e6])
@pytest.mark.parametrize("step", [1e-3, 1e-6, 1e-9])
@pytest.mark.parametrize("wide", [False, True])
def test_a_fast_uniform_motion(sums, forces, boost, step, wide):
    """Differences far below the velocities themselves, down to what the velocities
    still resolve."""
    h = 1.125 / 150
    pos, vel = _elements(9, 200, h, 0.05)
    vel = np.ascontiguousarray(boost * (1 + np.arange(3)[None, :, None]) + step * vel)
    for half_dt in (0.0, 1e-3 * h / boost):
        taken, _, fixed, fp64, size = sums(pos, vel, half_dt, wide)
        assert taken.all()
        _no_further_off(fixed, fp64, size, range(10))
    scal = np.tile([1 / (12 * h ** 3), -30 * h * h, -10.0], (200, 1))
    taken, fixed, fp64, size = forces(pos, vel, scal, wide)
    assert taken.all()
    _no_further_off(fixed, fp64, size, range(3))


@pytest.mark.parametrize("away", [12, 20, 24, 28, 32, 40])
@pytest.mark.parametrize("axes", [(0,), (1, 2), (0, 1, 2)])
@pytest.mark.parametrize("wide", [False, True])
def test_a_mesh_far_from_the_origin(sums, forces, away, axes, wide):
    """2^away spacings from it, along some axes; the extents are known exactly there too."""
    h = 1.125 / 150
    pos, vel = _elements(10, 200, h, 0.05)
    pos -= h * np.floor(pos[:, :, :1] / h)
    pos[:, list(axes)] += h * 2.0 ** away
    taken, _, fixed, fp64, size = sums(pos, vel, 1e-4 * h, wide)
    assert taken.all()
    _no_further_off(fixed, fp64, size, range(10))
    scal = np.stack([1 / _volume12(pos), np.full(200, -30 * h * h), np.full(200, -10.0)], 1)
    taken, fixed, fp64, size = forces(pos, vel, scal, wide)
    assert taken.all()
    _no_further_off(fixed, fp64, size, range(3))


def test_exact_zeros_stay_zeros(sums):
    """Velocities of zeros of both signs, and a flow whose divergence is exactly
    zero in doubles (compression along one axis as expansion along another, on
    either side of rest): the sums are zeros, as in FP64. A divergence that is not
    would set a time constraint (src/domain.jl:2964-3014)."""
    h = 0.125
    pos = np.ascontiguousarray(h * (np.array([[[2.0], [3.0], [5.0]]]) + CUBE))
    r = np.random.default_rng(3)
    vel = np.where(r.random((200, 3, 8)) < 0.5, 0.0, -0.0)
    many = np.ascontiguousarray(np.broadcast_to(pos, (200, 3, 8)))
    taken, want, fixed, _, _ = sums(many, np.ascontiguousarray(vel), 1e-6)
    assert taken.all() and not want[:, 5:9].any() and not fixed[:, 5:9].any()
    for i in range(3):
        j, k = (i + 1) % 3, (i + 2) % 3
        for a, b in ((1.0, 0.0), (0.75, 0.25), (0.1, 0.2)):
            v = np.zeros((1, 3, 8))
            v[0, i] = np.where(CUBE[i] > 0, a, -a)  # a - (-a)
            v[0, j] = np.where(CUBE[j] > 0, b, b + 2 * a)
            v[0, k] = -0.0
            taken, want, fixed, fp64, _ = sums(pos, v, 0.0)
            assert taken.all()
            if (b + 2 * a) - b == 2 * a:
                assert want[0, 8] == 0 and fp64[0, 8] == 0 and fixed[0, 8] == 0, (i, a, b)
            assert fixed[0, 5 + k] == 0


@pytest.mark.parametrize("h", [1.125 / 30, 1.125 / 150, 2.0 ** -7])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("squash", [1.0, 0.5, 0.2, 0.09, 1 / 25, 1 / 32])
def test_forces_of_thin_elements(forces, h, axis, squash):
    """The pure stress, the hourglass forces, and both."""
    pos, vel = _elements(4, 400, h, 0.02, squash, axis)
    r = np.random.default_rng(5)
    vi12 = 1 / (12 * h ** 3 * squash * r.uniform(0.95, 1.05, 400))
    for coef, s8 in ((0.0, -100.0), (-30.0 * h * h, 0.0), (-30.0 * h * h, -10.0)):
        scal = np.stack([vi12, np.full(400, coef), np.full(400, s8)], 1)
        taken, fixed, fp64, size = forces(pos, vel, scal)
        assert taken.all() if squash > 0.1 else taken.any()
        _no_further_off(fixed[taken], fp64[taken], size[taken], range(3))


def _slender(seed, n, size, thin, rotated):
    """Plates and needles (edges size and size * thin), jittered in their own
    coordinates, some distance from the origin, along the axes or turned."""
    r = np.random.default_rng(seed)
    e = CUBE + 0.03 * r.uniform(-1, 1, (n, 3, 8)) + np.floor(r.uniform(0, 50, (n, 3, 1)))
    few = r.integers(0, 3, n)
    many = r.random(n) < 0.5
    for i in range(n):
        for k in range(3):
            if (k == few[i]) == many[i]:
                e[i, k] *= thin
    if rotated:
        q = np.linalg.qr(r.standard_normal((n, 3, 3)))[0]
        q *= np.sign(np.linalg.det(q))[:, None, None]
        e = q @ e
    return np.ascontiguousarray(size * e), np.ascontiguousarray(r.uniform(-1, 1, (n, 3, 8)))


def _volume12(p):
    def d(a, b):
        return p[:, :, a] - p[:, :, b]
    t = ((d(3, 1) + d(7, 2), d(6, 3), d(2, 0)), (d(4, 3) + d(5, 7), d(6, 4), d(7, 0)),
         (d(1, 4) + d(2, 5), d(6, 1), d(5, 0)))
    return sum((u * np.cross(v, w)).sum(1) for u, v, w in t)


@pytest.mark.parametrize("size", [2.0 ** -90, 1e-9, 1e-5, 0.01, 1e13, 2.0 ** 90])
@pytest.mark.parametrize("thin", [1.0, 0.1, 1e-2, 1e-3])
@pytest.mark.parametrize("rotated", [False, True])
def test_the_kernels_range(sums, forces, size, thin, rotated):
    """Plates and needles along the axes, forces of turned ones, elements of any size."""
    pos, vel = _slender(6, 300, size, thin, rotated)
    ext = (pos.max(2) - pos.min(2)).min(1)
    taken, want, fixed, fp64, size_ = sums(pos, vel, 1e-3 * ext.min(), wide=True)
    assert taken.all() or (rotated and thin < 0.1)  # (turned ones are the kinematics' to 1/32 of their box)
    if taken.any():
        _no_further_off(fixed[taken], fp64[taken], size_[taken], range(10))
    scal = np.stack([1 / _volume12(pos), np.full(300, -1.0), np.full(300, -1 / size / size)], 1)
    taken, fixed, fp64, size_ = forces(pos, vel, scal, wide=True)
    assert taken.all()
    _no_further_off(fixed, fp64, size_, range(3))


def test_what_the_kernels_range_refuses(sums, forces):
    """Inverted, flat and non-finite elements, and extents beyond 2^100."""
    pos, vel = _slender(7, 8, 0.01, 1.0, True)
    pos[0] = pos[0, :, [4, 5, 6, 7, 0, 1, 2, 3]].T
    pos[1, :, 4:] = pos[1, :, :4]
    pos[2, 1, 3] = np.nan
    pos[3, 0, 7] = np.inf
    pos[4] *= 1e35
    pos[5] *= 1e-35
    vel[6, 2, 1] = np.inf
    scal = np.tile([1.0, -1.0, -1.0], (8, 1))
    assert sums(pos, vel, 1e-9, wide=True)[0].tolist() == [False] * 7 + [True]
    scal[:, 0] = 1 / 12e-6
    assert forces(pos, vel, scal, wide=True)[0].tolist() == [False] * 7 + [True]


def test_base_vectors_stay_in_bounds(lib):
    """Elements as distorted as they come, with volumes of state far from their own:
    three products of derivatives below 2^60 and modes below 2^62 over 2^64, and 2^58
    for gamma, are below 2^60; the sums over corners hold seven times that and no more."""
    r = np.random.default_rng(8)
    n = 40000
    e = CUBE + r.uniform(0, 0.5, (n, 1, 1)) * r.choice([-1, 1], (n, 3, 8)) * r.uniform(0.5, 1, (n, 3, 8))
    e[:, 2] *= 10 ** r.uniform(-3, 0, (n, 1))
    q = np.linalg.qr(r.standard_normal((n, 3, 3)))[0]
    q *= np.sign(np.linalg.det(q))[:, None, None]
    turned = r.random(n) < 0.6
    e[turned] = (q @ e)[turned]
    pos = np.ascontiguousarray(0.01 * e)
    w = _volume12(pos)
    pos, w = np.ascontiguousarray(pos[w > 0]), w[w > 0]
    n = len(w)
    vel = np.ascontiguousarray(r.choice([-1.0, 1.0, 0.99], (n, 3, 8)))
    scal = np.ascontiguousarray(np.stack([10 ** r.uniform(-1, 3, n) / w, np.full(n, -1.0), np.zeros(n)], 1))
    largest = np.zeros(n)
    lib.check_base(n, *(a.ctypes.data_as(ctypes.c_void_p) for a in (pos, vel, scal, largest)))
    assert (largest > 0).mean() > 0.5 and largest.max() < 2.0 ** 60
