"""A gradient does not depend on how its run is cut into segments: the taped cycles
(which the recompute repeats) have the bits of the untaped ones, also without
hourglass forces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STATE = ("e", "p", "q", "v", "ss", "x", "y", "z", "xd", "yd", "zd")


@pytest.mark.parametrize("mode", [0, 7])
@pytest.mark.parametrize("hgcoef", [3.0, 0.0, -1.0])
def test_segments_of_a_gradient(gpu_lib, mode, hgcoef):
    L = gpu_lib
    out = []
    for every in (24, 7, 3):
        g = L.Domain(L.LuleshProblem(nx=6, mode=mode))
        L.run(g, 10)
        g.hgcoef = hgcoef
        adj = L.Adjoint(g, checkpoint_every=every)
        loss = adj.gradient(24)
        out.append([loss, adj.result.grad_hgcoef] + [adj.grad(f) for f in STATE] + [g.field(f) for f in STATE])
        adj.close()
        g.close()
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)
