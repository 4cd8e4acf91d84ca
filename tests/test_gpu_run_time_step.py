"""The device run loop's time step beside the forces (one kernel) against the
per-step calls, which launch them one after the other: bitwise the same states,
the same errors, and no error from a cycle that does not take place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STATE = ("x", "y", "z", "xd", "yd", "zd", "e", "p", "q", "v", "ss")


def make(L, nx, mode=0):
    return L.Domain(L.LuleshProblem(nx=nx, nr=1, mode=mode))


@pytest.mark.parametrize("nx,cycles", [(1, 2), (2, 3), (3, 17), (6, 33)])
@pytest.mark.parametrize("mode", [0, 7])
def test_run_equals_stepping(gpu_lib, nx, cycles, mode):
    L = gpu_lib
    a, b = make(L, nx, mode), make(L, nx, mode)
    L.run(a, cycles)
    while b.cycle < cycles and b.time < b.stoptime:
        L.timeIncrement(b)
        L.lagrangeLeapFrog(b)
    assert (a.cycle, a.time, a.deltatime) == (b.cycle, b.time, b.deltatime)
    for f in STATE:
        assert np.array_equal(a.field(f), b.field(f)), f


@pytest.mark.parametrize("nx", [2, 5])
@pytest.mark.parametrize("kind", ["v", "x"])
def test_errors_of_the_forces(gpu_lib, nx, kind):
    L = gpu_lib

    def broken():
        g = make(L, nx)
        if kind == "v":
            v = g.field("v")
            v[-1] = -1.0
            g.set_field("v", v)
        else:
            x = g.field("x")
            g.set_field("x", x.max() - x)  # inverted elements
        return g
    # a run that takes no cycle raises nothing and leaves the state as it was
    g = broken()
    before = {f: g.field(f) for f in STATE}
    stoptime, g.stoptime = g.stoptime, g.time
    L.run(g, 5)
    assert g.cycle == 0
    for f in STATE:
        assert np.array_equal(g.field(f), before[f]), f
    # the next one does raise, what the per-step calls raise
    g.stoptime = stoptime
    with pytest.raises(L.LuleshError) as run_error:
        L.run(g, 5)
    h = broken()
    L.timeIncrement(h)
    with pytest.raises(L.LuleshError) as step_error:
        L.lagrangeLeapFrog(h)
    assert str(run_error.value) == str(step_error.value)
    assert g.cycle == h.cycle and g.time == h.time


def test_more_problems_than_one_block_steps(gpu_lib):
    """96 problems' time steps to a block: 95, 96, 97 and 200 problems."""
    L = gpu_lib
    single = {}
    for nx in (1, 2, 3):
        g = make(L, nx)
        L.run(g, 6)
        single[nx] = (g.time, g.field("e"))
    for n in (95, 96, 97, 200):
        ens = L.Ensemble([{"nx": 1 + i % 3, "nr": 1} for i in range(n)])
        ens.run(6)
        for i in (0, 1, 94, n - 2, n - 1):
            time, e = single[1 + i % 3]
            assert ens.scalars(i)["time"] == time and np.array_equal(ens.field(i, "e"), e), (n, i)
        ens.close()
