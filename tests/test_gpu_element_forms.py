"""Blocks that mix elements of the fixed-point form with elements it does not take
(the FP64 form of lulesh_element_fp64.cuh), against the CPU oracle at the parity
bar: forces of elements whose pressure or sound speed is below the numbers the
fixed-point form takes, kinematics of elements whose corners move by 0.3 of an edge
in half a step. And meshes of slender and of very small elements, which the
fixed-point form takes."""
import numpy as np
import pytest

from test_gpu_fixed_point import _volume
from test_gpu_parity import AUX_F64, STEP_F64, assert_fields, assert_scalars, pair

pytestmark = pytest.mark.gpu


def _both(g, o, state, dt):
    for f, v in state.items():
        g.set_field(f, v)
        o.set_field(f, v)
    for s in ("deltatime", "dtfixed"):
        setattr(g, s, dt)
        o.set(s, dt)


def _steps(L, g, o, n):
    for step in range(n):
        L.timeIncrement(g)
        o.time_increment()
        L.lagrangeLeapFrog(g)
        assert o.lagrange_leapfrog() == 0
        assert_scalars(g, o)
        assert_fields(g, o, STEP_F64 + AUX_F64, where=f"step {step}")


@pytest.mark.parametrize("nx", [2, 7])
@pytest.mark.parametrize("mode", [0, 7])
def test_mixed_forms_match_oracle(gpu_lib, oracle_mod, mode, nx):
    rng = np.random.default_rng(0xF0 + nx)
    g, o = pair(gpu_lib, oracle_mod, nx, mode=mode, keep_aux=True)
    E, N = g.numElem, g.numNode
    h, dt = 1.125 / nx, 0.05
    p = np.stack([g.field(k) for k in "xyz"])
    plane = np.rint(p[0] / h).astype(int)
    p += 0.02 * h * rng.uniform(-1, 1, p.shape) * (p > 0)
    nl = g.field("nodelist").reshape(E, 8).T
    state = dict(zip("xyz", p))
    state |= {"v": _volume(p, nl) / g.field("volo"), "e": rng.uniform(0.01, 0.1, E),
              "p": np.where(rng.random(E) < 0.2, 1e-130, rng.uniform(1e-3, 1e-2, E)), "q": np.zeros(E),
              "ss": np.where(rng.random(E) < 0.2, 1e-130, rng.uniform(1e-3, 1e-2, E))}
    # every third layer of elements stretched by 0.6 of its width in the step
    stretch = np.concatenate([[0.0], np.cumsum(np.where(np.arange(nx) % 3 == 0, 0.6, 0.0))])
    state["xd"] = h / dt * stretch[plane] + rng.normal(0, 0.01, N)
    state["yd"], state["zd"] = rng.normal(0, 0.01, N), rng.normal(0, 0.01, N)
    _both(g, o, state, dt)
    _steps(gpu_lib, g, o, 2)
    g.close()
    o.close()


@pytest.mark.parametrize("scale", [(1, 1, 1 / 200), (1, 1 / 80, 1 / 80), (1e-6, 1e-6, 1e-6), (1e-4, 1e-6, 1e-4)])
@pytest.mark.parametrize("mode", [0, 7])
def test_slender_and_small_meshes_match_oracle(gpu_lib, oracle_mod, mode, scale):
    nx = 5
    rng = np.random.default_rng(0xF8)
    g, o = pair(gpu_lib, oracle_mod, nx, mode=mode, keep_aux=True)
    E, N = g.numElem, g.numNode
    h = 1.125 / nx
    p = np.stack([g.field(k) for k in "xyz"])
    p += 0.03 * h * rng.uniform(-1, 1, p.shape) * (p > 0)
    p *= np.array(scale)[:, None]
    nl = g.field("nodelist").reshape(E, 8).T
    vol, thin = _volume(p, nl), 1.125 / nx * min(scale)
    nodal = np.bincount(nl.reshape(-1), np.tile(vol / 8, 8), N)
    state = dict(zip("xyz", p))
    state |= {"volo": vol, "elemMass": vol, "nodalMass": nodal, "v": np.ones(E), "e": rng.uniform(1, 200, E),
              "p": rng.uniform(1, 100, E), "q": rng.uniform(0, 5, E), "ss": rng.uniform(1, 10, E)}
    for f in ("xd", "yd", "zd"):
        state[f] = rng.normal(0, 0.5, N)
    _both(g, o, state, 1e-5 * thin)
    _steps(gpu_lib, g, o, 2)
    g.close()
    o.close()
