"""The force and kinematics kernels on meshes whose blocks mix elements of the
fixed-point form with elements of the FP64 form (thin ones), against the CPU
oracle at the parity bar: every step field and kept auxiliary field to 1e-8
with the parity floors.

Layers of the mesh are squashed along z to 1/250 and 1/1000 of their height
(below 1/256 of its bounding box an element is never taken, above 1/32 always;
1/100 lies between), with sheared and jittered corners, so blocks of 32
elements hold both kinds and the ragged last block does too.
"""
import numpy as np
import pytest

from conftest import rel_err  # noqa: F401  (the parity module's helpers use it)
from test_gpu_parity import AUX_F64, STEP_F64, assert_fields, assert_scalars, pair

pytestmark = pytest.mark.gpu


def _volume(p, nl):
    c = p[:, nl]

    def d(a, b):
        return c[:, a] - c[:, b]
    t = ((d(3, 1) + d(7, 2), d(6, 3), d(2, 0)), (d(4, 3) + d(5, 7), d(6, 4), d(7, 0)),
         (d(1, 4) + d(2, 5), d(6, 1), d(5, 0)))
    return sum((u * np.cross(v, w, axis=0)).sum(0) for u, v, w in t) / 12.0


@pytest.mark.parametrize("nx,squash,seed", [(7, 1 / 250, 0xE0), (7, 1 / 1000, 0xE1), (7, 1 / 100, 0xE2), (2, 1 / 1000, 0xE3)])
@pytest.mark.parametrize("mode", [0, 7])
def test_thin_and_ordinary_elements_match_oracle(gpu_lib, oracle_mod, mode, nx, squash, seed):
    rng = np.random.default_rng(seed)
    g, o = pair(gpu_lib, oracle_mod, nx, mode=mode, keep_aux=True)
    E, N = g.numElem, g.numNode
    h = 1.125 / nx
    p = np.stack([g.field(k) for k in "xyz"])
    layer = np.rint(p[2] / h).astype(int)
    heights = np.where(np.arange(nx) % 3 == 1, squash, 1.0) * h
    p[2] = np.concatenate([[0.0], np.cumsum(heights)])[layer]
    inside = (p[0] > 0) & (p[1] > 0) & (layer > 0)
    p[0] += inside * h * (0.02 * rng.uniform(-1, 1, N) + 0.1 * p[1])
    p[1] += inside * h * 0.02 * rng.uniform(-1, 1, N)
    p[2] += inside * h * 0.1 * squash * rng.uniform(-1, 1, N)
    nl = g.field("nodelist").reshape(E, 8).T
    state = dict(zip("xyz", p))
    state |= {"v": _volume(p, nl) / g.field("volo"), "e": rng.uniform(1e2, 2e4, E), "p": rng.uniform(0, 1e3, E),
              "q": rng.uniform(0, 50, E) * (rng.random(E) < 0.3), "ss": rng.uniform(1, 50, E)}
    assert state["v"].min() > 0
    for f in ("xd", "yd", "zd"):
        state[f] = rng.normal(0, 0.5, N) * (rng.random(N) < 0.8)
    for f, v in state.items():
        g.set_field(f, v)
        o.set_field(f, v)
    for s in ("deltatime",):
        setattr(g, s, 1e-9)
        o.set(s, 1e-9)
    for step in range(2):
        gpu_lib.timeIncrement(g)
        o.time_increment()
        gpu_lib.lagrangeLeapFrog(g)
        assert o.lagrange_leapfrog() == 0
        assert_scalars(g, o)
        assert_fields(g, o, STEP_F64 + AUX_F64, where=f"step {step}")
    g.close()
    o.close()


@pytest.mark.parametrize("nx", [2, 3, 6])
@pytest.mark.parametrize("mode", [0, 7])
def test_adjoint_forms_agree(gpu_lib, mode, nx):
    """The reverse sweep is linear in its seeds, and seeds of 2^-700 or 2^480
    are outside what its integer sums take (2^-400 to 2^400): the FP64 form's
    gradients, scaled back exactly, against the integer form's. 2 cycles of 8
    dependent sums of at most 64 terms, rounded to 2^-53 of partial sums up to
    2^8 times the largest gradient of the field."""
    tol = 2 * 8 * 64 * 2.0 ** -53 * 2 ** 8
    rng = np.random.default_rng(0xE8 + nx)
    fields = ("x", "y", "z", "xd", "yd", "zd", "e", "p", "q", "v", "ss")
    out = []
    state = seeds = None
    for scale in (0, -700, 480):
        g = gpu_lib.Domain(gpu_lib.LuleshProblem(nx=nx, mode=mode))
        if state is None:
            state = g.e + 1e4 * (1.0 + rng.random(g.numElem))
            seeds = {f: rng.standard_normal(g.field(f).size) * (rng.random(g.field(f).size) < 0.7) for f in fields}
        g.e = state
        gpu_lib.run(g, 3)
        adj = gpu_lib.Adjoint(g, checkpoint_every=1)
        for f in fields:
            adj.set_seed(f, seeds[f] * 2.0 ** scale)
        adj.gradient(2)
        out.append({f: adj.grad(f) * 2.0 ** -scale for f in fields})
        adj.close()
    for other in out[1:]:
        for f in fields:
            assert np.abs(other[f] - out[0][f]).max() <= tol * np.abs(out[0][f]).max(), f
