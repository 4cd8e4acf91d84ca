"""The reverse sweep's fixed-point crosses where one coordinate's adjoints are far
above the others': the component along it is made of the others alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "z", "xd", "yd", "zd")


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("ratio", [-20, -40])
def test_adjoints_along_one_axis(gpu_lib, axis, ratio):
    """Constant pressures (pmin above every other), no viscosity, no hourglass
    forces: what positions do to later velocities goes through the faces' area
    vectors only, and the component along the axis of the large seeds comes from
    the small ones. Seeds scaled by 2^-700 take the crosses in doubles
    (test_adjoint_forms_agree); each field against its own largest value, at the
    bound derived there."""
    tol = 2 * 8 * 64 * 2.0 ** -53 * 2 ** 8
    L, rng = gpu_lib, np.random.default_rng(0xAD + axis)
    out = []
    state = seeds = None
    for scale in (0, -700):
        g = L.Domain(L.LuleshProblem(nx=4, mode=7))
        E, N = g.numElem, g.numNode
        if state is None:
            state = {"e": rng.uniform(0.5, 1, E), "p": np.full(E, 100.0), "q": np.zeros(E), "ss": np.ones(E)}
            state |= {f: rng.normal(0, 0.3, N) for f in ("xd", "yd", "zd")}
            seeds = {f: rng.standard_normal(N) for f in ("xd", "yd", "zd")}
            for k, f in enumerate(seeds):
                if k != axis:
                    seeds[f] *= 2.0 ** ratio
        for s, v in {"pmin": 100.0, "hgcoef": 0.0, "qlc_monoq": 0.0, "qqc_monoq": 0.0, "u_cut": 0.0, "dtfixed": 1e-6,
                     "deltatime": 1e-6}.items():
            setattr(g, s, v)
        for f, v in state.items():
            g.set_field(f, v)
        adj = L.Adjoint(g, checkpoint_every=4)
        for f, w in seeds.items():
            adj.set_seed(f, w * 2.0 ** scale)
        adj.gradient(3)
        out.append({f: adj.grad(f) * 2.0 ** -scale for f in FIELDS})
        adj.close()
        g.close()
    along = "xyz"[axis]
    assert np.abs(out[1][along]).max() < 2.0 ** (ratio / 2) * max(np.abs(out[1][f]).max() for f in "xyz")
    for f in FIELDS:
        assert np.abs(out[0][f] - out[1][f]).max() <= tol * np.abs(out[1][f]).max(), f
