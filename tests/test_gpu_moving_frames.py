"""A mesh far from the origin and in fast uniform motion: forces are those of the same
mesh at rest beside the origin, and the velocity gradients those of extended
precision. (The oracle's own hourglass sums cancel there.) Positions and velocities are
multiples of powers of two, so that the shift and the boost are exact.

Bounds, of the element arithmetic: forces of a corner 2^-48 of |s8| E^2 +
|coefficient| dV, eight corners in either run; a velocity gradient 2^-49 of
E^2 dV / volume, with the volume's 2^-47 and the quotient's rounding below 2^-46."""
import numpy as np
import pytest

from test_gpu_fixed_point import _volume

pytestmark = pytest.mark.gpu

SHIFT, BOOST = 2.0 ** 26, 2.0 ** 30


def _run(L, nx, mode, shift, boost):
    g = L.Domain(L.LuleshProblem(nx=nx, mode=mode, keep_aux=True))
    rng = np.random.default_rng(0xFA)
    E, N, h = g.numElem, g.numNode, 1.125 / nx
    p = np.stack([g.field(k) for k in "xyz"]) + 0.03 * h * rng.uniform(-1, 1, (3, N))
    p = np.round(p * 2.0 ** 26) / 2.0 ** 26
    u = np.round(rng.uniform(-1, 1, (3, N)) * 2.0 ** 20) / 2.0 ** 20
    nl = g.field("nodelist").reshape(E, 8).T
    state = {"v": _volume(p, nl) / g.field("volo"), "e": rng.uniform(1, 10, E), "p": rng.uniform(1, 10, E),
             "q": rng.uniform(0, 1, E), "ss": rng.uniform(1, 10, E)}
    state |= dict(zip("xyz", p + shift)) | dict(zip(("xd", "yd", "zd"), u + boost))
    for f, v in state.items():
        g.set_field(f, v)
    g.deltatime = g.dtfixed = 2.0 ** -60
    L.timeIncrement(g)
    L.lagrangeLeapFrog(g)
    out = {f: g.field(f) for f in ("fx", "fy", "fz", "x", "y", "z", "xd", "yd", "zd", "delv_xi", "delv_eta",
                                   "delv_zeta", "vnew", "volo", "elemMass")}
    g.close()
    return p, nl, state, out


@pytest.mark.parametrize("nx", [2, 7])
@pytest.mark.parametrize("mode", [0, 7])
@pytest.mark.parametrize("shift,boost", [(SHIFT, 0.0), (0.0, BOOST), (SHIFT, BOOST)])
def test_forces_and_gradients_in_a_moving_frame(gpu_lib, mode, nx, shift, boost):
    p, nl, state, rest = _run(gpu_lib, nx, mode, 0.0, 0.0)
    _, _, _, moved = _run(gpu_lib, nx, mode, shift, boost)
    ext = np.ptp(p[:, nl], axis=1).max(0)
    coef = 3.0 * 0.01 * state["ss"] * rest["elemMass"] / np.cbrt(state["v"] * rest["volo"])
    corner = 2.0 ** -48 * ((state["p"] + state["q"]) / 8 * ext ** 2 + coef * 2)
    for f in ("fx", "fy", "fz"):
        assert np.abs(moved[f] - rest[f]).max() <= 16 * corner.max(), f

    x, v = (np.stack([moved[k] for k in names])[:, nl].astype(np.longdouble)
            for names in (("x", "y", "z"), ("xd", "yd", "zd")))  # [coordinate][corner][element], end of the step
    signs = np.array([[-1, 1, 1, -1, -1, 1, 1, -1], [-1, -1, 1, 1, -1, -1, 1, 1], [-1, -1, -1, -1, 1, 1, 1, 1]])
    edge, diff = (np.einsum("ac,kce->ake", signs, a - a[:, :1]) / 4 for a in (x, v))
    vol = moved["volo"] * moved["vnew"]
    ext, dv = np.ptp(x, axis=1).max(0), np.ptp(v, axis=1).max(0)
    for a, f in enumerate(("delv_xi", "delv_eta", "delv_zeta")):
        area = np.cross(edge[(a + 1) % 3], edge[(a + 2) % 3], axis=0)
        want = (area * diff[a]).sum(0) / vol
        off = np.abs(moved[f] - want) / (ext ** 2 * dv / vol)
        assert off.max() <= 2.0 ** -46, f
