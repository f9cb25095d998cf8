"""The FP64 translation by sibling families (k_m2l_group, schedule bit 0 set)
against the per-box kernel (bit 0 clear): the same sums in another order, so
products agree to the rounding of sums of at most 189 terms (189 x 2.2e-16 =
4e-14, here 1e-13), over families of one to eight siblings, lists longer than a
staged batch of 32, grids that are not a multiple of the 16-direction run,
boxes with empty lists under both rules, and the transposed product."""
import numpy as np
import pytest

from mlfma_b200 import MLFMA, inputs

pytestmark = pytest.mark.gpu
PW = inputs.PlaneWave()


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def cvec(n, seed):
    r = np.random.default_rng(seed)
    return r.standard_normal(n) + 1j * r.standard_normal(n)


def clusters(n, seed):
    """A dense cluster and a few far ones: single-box families, empty lists."""
    r = np.random.default_rng(seed)
    c = np.array([[-1.5, -1.5, -1.5], [1.6, 1.4, 1.5], [1.4, -1.6, 0.2]])
    k = np.minimum(r.integers(0, 8, n), 2)
    pos = c[k] + r.uniform(-0.2, 0.2, (n, 3))
    return inputs.Dipoles(pos=pos, mom=np.tile([0.0, 0.0, 1.0], (n, 1)))


CASES = {
    "cloud_full_siblings": (lambda: inputs.make_dipoles(6000, seed=3), dict(max_node_srcs=4, max_level=4)),
    "cloud_two_levels": (lambda: inputs.make_dipoles(8192, seed=1), dict(max_node_srcs=64)),
    "one_level": (lambda: inputs.make_dipoles(600, seed=1), dict(max_node_srcs=64)),
    "clusters": (lambda: clusters(900, 5), dict(max_node_srcs=16)),
    "sphere": (lambda: inputs.make_icosphere(4, radius=1.13), dict(max_node_srcs=54, root_leng=2.26)),
}


@pytest.mark.parametrize("case", list(CASES))
@pytest.mark.parametrize("ref_compat", [0, 1])
def test_families_match_per_box_kernel(cuda_device, case, ref_compat):
    make, cfg = CASES[case]
    g = make()
    build = MLFMA.rwg if case == "sphere" else MLFMA.dipoles
    ys = {}
    for sched in (0, 1):
        op = build(g, PW, ref_compat=ref_compat, **cfg).setup()
        op.set_schedule(sched)
        ys[sched] = [op.matvec(cvec(op.n, s)) for s in (1, 2, 3)]
        if not ref_compat:
            ys[sched].append(op.matvec_adjoint(cvec(op.n, 4)))
        op.close()
    for a, b in zip(ys[1], ys[0]):
        assert rel(a, b) <= 1e-13
