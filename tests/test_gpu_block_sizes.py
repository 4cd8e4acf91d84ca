"""The block sizes that change launches (node_block, mat_block; the default follows the
mesh) give bitwise the same states and gradients, also when they change in the middle
of a run, on meshes below and above eight blocks per SM."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STATE = ["e", "p", "q", "v", "ss", "x", "y", "z", "xd", "yd", "zd"]
SIZES = [{"node_block": 128, "mat_block": 64}, {"node_block": 512, "mat_block": 256}, {"node_block": 256, "mat_block": 128}]


def _same(a, b):
    for f in STATE + ["vdov", "arealg", "delv"]:
        assert np.array_equal(a.field(f), b.field(f)), f
    for s in ("time", "deltatime", "dtcourant", "dthydro", "cycle"):
        assert getattr(a, s) == getattr(b, s), s


@pytest.mark.parametrize("nx,mode,tp", [(1, 0, 1), (12, 0, 1), (12, 7, 1), (70, 0, 1), (6, 7, 2)])
def test_domain(gpu_lib, nx, mode, tp):
    L = gpu_lib
    a = L.Domain(L.LuleshProblem(nx=nx, mode=mode, blocks_per_edge=tp))
    L.run(a, 40)
    b = L.Domain(L.LuleshProblem(nx=nx, mode=mode, blocks_per_edge=tp))
    for k, sizes in enumerate(SIZES):
        b.set_tuning(**sizes)
        assert {n: b.tuning()[n] for n in sizes} == sizes
        L.run(b, 10 * (k + 1))
    while b.cycle < a.cycle:  # (a's run may have reached stoptime)
        L.timeIncrement(b)
        L.lagrangeLeapFrog(b)
    _same(a, b)


def test_ensemble(gpu_lib):
    L = gpu_lib
    inst = [{"nx": 5, "nr": 11}, {"nx": 9, "nr": 1, "hgcoef": 2.2}, {"nx": 3, "einit": 1e5}]
    a = L.Ensemble(inst)
    a.run(40)
    for sizes in SIZES:
        b = L.Ensemble(inst)
        b.set_tuning(**sizes)
        b.run(25)
        b.set_tuning(**SIZES[0])
        b.run(40)
        for i in range(len(inst)):
            for f in STATE:
                assert np.array_equal(a.field(i, f), b.field(i, f)), (i, f)


def test_adjoint(gpu_lib):
    L = gpu_lib
    res = []
    for sizes in SIZES:
        g = L.Domain(L.LuleshProblem(nx=8))
        L.run(g, 5)
        g.set_tuning(**sizes)
        adj = L.Adjoint(g, checkpoint_every=6)
        adj.gradient(25)
        g.set_tuning(**SIZES[0])
        loss = adj.gradient(20)
        res.append([loss, adj.result.grad_hgcoef] + [adj.grad(f) for f in STATE] + [g.field("e")])
        adj.close()
        g.close()
    for other in res[1:]:
        for x, y in zip(res[0], other):
            assert np.array_equal(x, y)
