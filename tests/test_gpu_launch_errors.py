"""Solves report a kernel launch that was refused, and only their own: an error
that an earlier call of the thread left behind (a setup on a device that is not
there) is not a later solve's."""
import numpy as np
import pytest

from mlfma_b200 import MLFMA, inputs
from mlfma_b200._lib import MlfmaError

pytestmark = pytest.mark.gpu
PW = inputs.PlaneWave()


@pytest.mark.parametrize("precision", [0, 1])
def test_earlier_error_is_not_the_solves(cuda_device, precision):
    d = inputs.make_dipoles(700, seed=2)
    kw = dict(ref_compat=0, self_terms=1, precision=precision, max_rhs=2)
    op = MLFMA.dipoles(d, PW, **kw).setup()
    b = op.rhs()
    want, _ = op.solve(b, max_iter=3, tol=1e-14, restart=3)
    wants, _ = op.solve_multi(np.stack([b, 2 * b]), max_iter=3, tol=1e-14, restart=3)
    for solve, w in ((lambda: op.solve(b, max_iter=3, tol=1e-14, restart=3)[0], want),
                     (lambda: op.solve_multi(np.stack([b, 2 * b]), max_iter=3, tol=1e-14, restart=3)[0], wants)):
        with pytest.raises(MlfmaError):
            MLFMA.dipoles(d, PW, device=4096, **kw).setup()
        assert np.array_equal(solve(), w)
    op.close()
