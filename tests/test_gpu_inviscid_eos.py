"""The EOS of elements without viscosity, whose sound speed is formed for q only
where it might not be finite: a mesh at rest with energies on both sides of the
bound (2^300) against the CPU oracle. An energy passes through at most 20
roundings without cancellation: 1e-14."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ENERGIES = [0.0, 1e-40, 1e-3, 1.0, 3.9e7, 2.0 ** 299, 2.0 ** 300, 2.0 ** 301, 1e150, -1.0]


@pytest.mark.parametrize("nx", [1, 3, 6])
@pytest.mark.parametrize("reps", [False, True])
def test_energies_at_rest_match_oracle(gpu_lib, oracle_mod, nx, reps):
    L = gpu_lib
    g = L.Domain(L.LuleshProblem(nx=nx, nr=3, cost=2, region_reps=reps))
    o = oracle_mod.OracleDomain(nx, nr=3)
    e = np.resize(np.array(ENERGIES), g.numElem)
    g.e = e
    o.set_field("e", e)
    L.timeIncrement(g)
    L.lagrangeLeapFrog(g)
    o.time_increment()
    assert o.lagrange_leapfrog() == 0
    for f in ("e", "p", "q", "ss", "v"):
        a, b = g.field(f), o.field(f)
        assert np.all(np.abs(a - b) <= 1e-14 * np.abs(b)), (f, a, b)
