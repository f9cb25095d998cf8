"""A mixed operator tuned in complex float, and its FP64 far field, which runs the
same launch shapes with elements twice as large: on a 58 x 116 grid two column
pairs of the many-rhs anterpolation fit the one and not the other.  The FP64
residual that a refined or flexible solve reports is that of the FP64 operator
(products of some thousand terms in another order: 1e-12 of |A| |x|, a few times
|b| here; 1e-10)."""
import numpy as np
import pytest

from mlfma_b200 import MLFMA, inputs

pytestmark = pytest.mark.gpu
PW = inputs.PlaneWave()


def surface(n, radius, seed):
    v = np.random.default_rng(seed).standard_normal((n, 3))
    return inputs.Dipoles(pos=radius * v / np.linalg.norm(v, axis=1)[:, None], mom=np.tile([1.0, 0.0, 0.0], (n, 1)))


@pytest.mark.parametrize("kind", [dict(refine=True), dict(flexible=True, inner_iters=2)])
def test_tuned_mixed_solve_reports_its_fp64_residual(cuda_device, kind):
    cfg = dict(ref_compat=0, self_terms=1, max_node_srcs=30, root_leng=16.0)
    op = MLFMA.dipoles(surface(1200, 7.99, 8), PW, precision=1, max_rhs=4, **cfg).setup()
    op64 = MLFMA.dipoles(surface(1200, 7.99, 8), PW, precision=0, **cfg).setup()
    op.autotune(1, reps=2)
    for _ in range(12):  # (a choice by timing: until it takes the wider tile, if it ever does)
        if op.autotune(4, reps=2)["multi_l2l_pairs"] == 2:
            break
    r = np.random.default_rng(3)
    B = r.standard_normal((4, op.n)) + 1j * r.standard_normal((4, op.n))
    X, infos = op.solve_multi(B, max_iter=4, tol=1e-12, restart=2, **kind)
    for c in range(4):
        true = np.linalg.norm(B[c] - op64.matvec(X[c])) / np.linalg.norm(B[c])
        assert abs(infos[c].true_residual - true) <= 1e-10, (c, infos[c].true_residual, true)
    op.close()
    op64.close()
