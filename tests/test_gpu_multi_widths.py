"""The many-right-hand-side product at the edges of its kernels' forms, column by
column against the one-vector product: GEMM tiles of 16 to 64 columns, blocks of
one to four translation directions, sibling groups of one to eight targets
(single boxes, a surface, a full cloud), and interpolations that take
neighbouring outputs together (six points) or one at a time (four and eight
points; a 58 x 116 grid, whose tile is too large).  Sums of some thousand terms in
another order: 1e-12 FP64; complex float 1e-5."""
import numpy as np
import pytest

from mlfma_b200 import MLFMA, inputs

pytestmark = pytest.mark.gpu
PW = inputs.PlaneWave()


def surface(n, radius, seed):
    v = np.random.default_rng(seed).standard_normal((n, 3))
    return inputs.Dipoles(pos=radius * v / np.linalg.norm(v, axis=1)[:, None], mom=np.tile([1.0, 0.0, 0.0], (n, 1)))


CASES = {
    "cloud": (lambda: inputs.make_dipoles(2500, seed=3), dict(max_node_srcs=8)),
    "surface": (lambda: surface(3000, 1.99, 4), dict(max_node_srcs=8)),
    "sparse": (lambda: inputs.make_dipoles(60, seed=5), dict(max_node_srcs=1)),
    "four_points": (lambda: surface(1500, 1.99, 6), dict(max_node_srcs=8, interp_order=2)),
    "eight_points": (lambda: surface(1500, 1.99, 7), dict(max_node_srcs=24, interp_order=4)),
    "large_grid": (lambda: surface(1200, 7.99, 8), dict(max_node_srcs=30, root_leng=16.0)),
}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case,widths", [("cloud", (2, 15, 16, 17, 33, 48, 64)), ("surface", (3, 21, 32, 49, 64)),
                                         ("sparse", (5, 64)), ("four_points", (18,)), ("eight_points", (18,)),
                                         ("large_grid", (4,))])
def test_columns_match_one_vector(cuda_device, case, widths, precision):
    make, cfg = CASES[case]
    op = MLFMA.dipoles(make(), PW, ref_compat=0, precision=precision, max_rhs=max(widths), **cfg).setup()
    r = np.random.default_rng(11)
    X = r.standard_normal((max(widths), op.n)) + 1j * r.standard_normal((max(widths), op.n))
    tol = 1e-12 if precision == 0 else 1e-5
    one = {c: op.matvec(X[c]) for nr in widths for c in {0, nr // 2, nr - 1}}
    for nr in widths:
        Y = op.matvec_multi(X[:nr])
        for c in {0, nr // 2, nr - 1}:
            assert np.linalg.norm(Y[c] - one[c]) <= tol * np.linalg.norm(one[c]), (nr, c)
    op.close()
