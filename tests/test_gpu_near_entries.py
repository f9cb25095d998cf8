"""A near-field entry that is not finite spoils the two sums it belongs to and no
other, in every near-field kernel: two dipoles 2e-110 apart (their entry holds
1/R^3), in one leaf (a packed self block) and on either side of the plane between
two leaves (a rectangular block with padding lanes)."""
import numpy as np
import pytest

from mlfma_b200 import MLFMA, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na,nb", [(40, 0), (7, 0), (33, 21), (9, 40)])
@pytest.mark.parametrize("at", [0, 3, 5])
def test_entry_stays_in_its_sums(cuda_device, na, nb, at):
    r = np.random.default_rng(na + nb)
    pos = np.concatenate([r.uniform(0.05, 0.45, (na, 3)), -r.uniform(0.05, 0.45, (nb, 3))])
    i, j = at, na + at if nb else at + 1
    pos[i], pos[j] = 1e-110, -1e-110 if nb else 3e-110
    n = na + nb
    d = inputs.Dipoles(pos=pos, mom=np.tile([1.0, 2.0, -0.5], (n, 1)))
    op = MLFMA.dipoles(d, inputs.PlaneWave(), max_node_srcs=max(na, nb) if nb else 64, self_terms=0, ref_compat=0).setup()
    x = r.standard_normal(n) + 1j * r.standard_normal(n)
    want = np.ones(n, bool)
    want[[i, j]] = False
    for kind in (2, 0):
        op.set_near_kernel(kind)
        assert np.array_equal(np.isfinite(op.matvec(x)), want), kind
    op.close()
