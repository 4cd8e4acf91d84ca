"""k_material discards Courant candidates that are certainly above the least so far
by a comparison in single precision (lulesh_courant.cuh, compiled for the host): no
candidate below it may be discarded, whatever the units of the problem."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("courant") / "courant.so")
    subprocess.run([os.environ.get("CXX") or shutil.which("g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off",
                    os.path.join(ROOT, "tests", "courant_check.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)

    def run(*cols):
        cols = [np.ascontiguousarray(np.broadcast_to(np.asarray(c, float), np.broadcast_shapes(*map(np.shape, cols)))) for c in cols]
        n = cols[0].size
        says, above = np.zeros(n, np.int32), np.zeros(n, np.int32)
        lib.check_courant(n, *(a.ctypes.data_as(ctypes.c_void_p) for a in (*cols, says, above)))
        return says.astype(bool), above.astype(bool)
    return run


def _candidate(a, s, v, q):
    t = 8 * np.abs(q) * a * np.where(v < 0, -v, 0)
    m = np.maximum(s, t)
    with np.errstate(all="ignore"):
        return a / (m * np.sqrt((s / m) ** 2 + (t / m) ** 2))


@pytest.mark.parametrize("decades", [3, 20, 45, 150])
def test_nothing_below_the_least_is_discarded(check, decades):
    """Operands over 10^-decades to 10^decades, the least around the candidate."""
    r = np.random.default_rng(decades)
    n = 200000
    a, s, v = (10 ** r.uniform(-decades, decades, n) for _ in range(3))
    s[: n // 4] = 0.0
    v *= np.where(r.random(n) < 0.7, -1, 1)
    q = np.where(r.random(n) < 0.5, 2.0, 10 ** r.uniform(-45, 45, n))
    c = _candidate(a, s, v, q)
    least = np.where(r.random(n) < 0.5, c * 10 ** r.uniform(-1e-3, 3, n), c * (1 + 10 ** r.uniform(-16, -2, n)))
    ok = np.isfinite(least) & (least > 0)
    says, above = check(a[ok], s[ok], v[ok], least[ok], q[ok])
    assert not np.any(says & ~above)


def test_small_and_large_units(check):
    """Areas whose square, and rates whose square, a float does not hold; a least
    below the float range."""
    says, above = check([1e-25, 1e18, 1e-30, 1e-40], [1.0, 1e-10, 1e10, 1.0], [-1e25, -1e-19, 1.0, -1e38],
                        [1e-26, 1e25, 1e-39, 1e-41], 2.0)
    assert not np.any(says & ~above), (says, above)


def test_ordinary_candidates_are_discarded(check):
    """Candidates 1e-3 above the least are not formed."""
    r = np.random.default_rng(1)
    n = 10000
    a, s, v = 10 ** r.uniform(-4, 1, n), 10 ** r.uniform(-3, 3, n), -(10 ** r.uniform(-3, 4, n))
    says, _ = check(a, s, v, _candidate(a, s, v, 2.0) / 1.001, 2.0)
    assert says.all()
