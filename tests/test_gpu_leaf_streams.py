"""Aggregation and disaggregation (k_s2m, k_l2t and their half-pattern forms) at
the edges of their work items, against the numpy oracle: leaves of one source, of
more than a block's run, counts that are not a multiple of the rows in flight;
rows shorter than a warp's run, longer than one, and leaf grids above the size
whose local pattern is staged in shared memory (4,232 directions, 135 KB).
Tolerances: FP64 sums of some thousand terms, 1e-12; complex float, 1e-5."""
import numpy as np
import pytest

from mlfma_b200 import MLFMA, inputs
from oracle import mlfma_oracle as O

pytestmark = pytest.mark.gpu
PW = inputs.PlaneWave()
CASES = {
    "single_sources": dict(n=40, side=3.9, root=4.0, leaf=1),
    "large_leaves": dict(n=4000, side=3.9, root=4.0, leaf=100),
    "three_levels": dict(n=1111, side=3.9, root=4.0, leaf=9),
    "unstaged_grid": dict(n=200, side=11.9, root=12.0, leaf=12),
}


@pytest.mark.parametrize("case", list(CASES))
@pytest.mark.parametrize("precision", [0, 1])
def test_leaf_stages_match_oracle(cuda_device, case, precision):
    c = CASES[case]
    d = inputs.make_dipoles(c["n"], side=c["side"], seed=17)
    op = MLFMA.dipoles(d, PW, precision=precision, max_node_srcs=c["leaf"], root_leng=c["root"]).setup()
    if case == "unstaged_grid":
        assert op.level_info(2)["nth"] * op.level_info(2)["nph"] * 32 > 72 * 1024
    r = np.random.default_rng(5)
    x = r.standard_normal(op.n) + 1j * r.standard_normal(op.n)
    y = op.matvec(x)
    op.close()
    ref = O.Oracle(O.DipoleSources(d.pos, d.mom, PW), root_leng=c["root"], max_node_srcs=c["leaf"]).matvec(x)
    assert np.linalg.norm(y - ref) <= (1e-12 if precision == 0 else 1e-5) * np.linalg.norm(ref)
