"""The near field applied four tiles to a warp (k_near_direct) at the edges of its
tiles, against every interaction evaluated directly (mlfma_dense_rows): one leaf
of n sources (a packed self block, by whole rows up to 32 and by column ranges
above), two leaves of uneven size (rectangular blocks of 1 to 70 columns), with
and without the diagonal.  Sums of at most 140 products: 140 x 2.2e-16 = 3e-14,
here 1e-12."""
import numpy as np
import pytest

from mlfma_b200 import MLFMA, inputs

pytestmark = pytest.mark.gpu
PW = inputs.PlaneWave()


def check(pos, self_terms, leaf):
    d = inputs.Dipoles(pos=np.ascontiguousarray(pos), mom=np.tile([1.0, 2.0, -0.5], (len(pos), 1)))
    op = MLFMA.dipoles(d, PW, max_node_srcs=leaf, self_terms=self_terms, ref_compat=0).setup()
    r = np.random.default_rng(9)
    x = r.standard_normal(op.n) + 1j * r.standard_normal(op.n)
    want = op.dense_rows(np.arange(op.n), x)
    for kind in (2, 0):
        op.set_near_kernel(kind)
        assert np.linalg.norm(op.matvec(x) - want) <= 1e-12 * np.linalg.norm(want), kind
    op.close()


@pytest.mark.parametrize("self_terms", [0, 1])
@pytest.mark.parametrize("n", [2, 7, 8, 31, 32, 33, 64, 65, 130])
def test_one_leaf(cuda_device, n, self_terms):
    check(np.random.default_rng(n).uniform(-0.4, 0.4, (n, 3)), self_terms, 200)


@pytest.mark.parametrize("na,nb", [(1, 1), (1, 70), (3, 33), (25, 24), (40, 41), (70, 9)])
def test_two_leaves(cuda_device, na, nb):
    r = np.random.default_rng(na + 100 * nb)
    a, b = r.uniform(0.05, 0.45, (na, 3)), -r.uniform(0.05, 0.45, (nb, 3))
    check(np.concatenate([a, b]), 1, max(na, nb))


@pytest.mark.parametrize("at", [0, 20, 39])
def test_not_finite_stays_where_it_belongs(cuda_device, at):
    # one x of NaN and one pair of sources in one place (an entry that is not
    # finite): exactly the sums that contain them are not finite
    r = np.random.default_rng(4)
    pos = r.uniform(-1, 1, (40, 3))
    d = inputs.Dipoles(pos=pos, mom=np.tile([1.0, 2.0, -0.5], (40, 1)))
    op = MLFMA.dipoles(d, PW, max_node_srcs=64, self_terms=0, ref_compat=0).setup()
    x = r.standard_normal(op.n) + 1j * r.standard_normal(op.n)
    x[at] = np.nan
    masks = []
    for kind in (2, 0):
        op.set_near_kernel(kind)
        masks.append(np.isfinite(op.matvec(x)))
    assert masks[0][at] and masks[0].sum() == 1  # (no self term: every other sum has it)
    assert np.array_equal(masks[0], masks[1])
    op.close()
    pos[at] = pos[(at + 7) % 40]
    op = MLFMA.dipoles(inputs.Dipoles(pos=pos, mom=d.mom), PW, max_node_srcs=64, self_terms=0, ref_compat=0).setup()
    x[at] = 1.0
    masks = []
    for kind in (2, 0):
        op.set_near_kernel(kind)
        masks.append(np.isfinite(op.matvec(x)))
    assert np.array_equal(masks[0], masks[1])
    op.close()
