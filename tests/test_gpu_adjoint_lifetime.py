"""A domain destroyed before its adjoints (which a garbage collector does in any
order): they can still be read and destroyed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_adjoints_outlive_their_domain(gpu_lib):
    L = gpu_lib
    g = L.Domain(L.LuleshProblem(nx=5))
    L.run(g, 5)
    first, second, third = (L.Adjoint(g, checkpoint_every=k) for k in (4, 9, 20))
    second.close()
    first.gradient(9)
    third.gradient(3)
    before = first.grad("e")
    g.close()
    assert np.array_equal(first.grad("e"), before)
    for call in (lambda: first.gradient(2), first.loss, lambda: third.set_overlap(0)):
        with pytest.raises(L.LuleshError):
            call()
    third.close()
    first.close()
    # another domain in the freed memory is not touched by what is left
    h = L.Domain(L.LuleshProblem(nx=5))
    adj = L.Adjoint(h, checkpoint_every=4)
    adj.gradient(9)
    adj.close()
    h.close()
