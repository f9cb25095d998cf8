"""The FP64 translation by sibling families (k_m2l_group) where it can go wrong, on
levels that are known to run it: enough (pair, direction)s for families, boxes whose
list 2 is empty, single boxes and families of every size, under both rules for empty
lists (three products, the second and third from what the first left) and
transposed; against the per-box kernel.  The same sums of at most 189 terms in
another order: 189 x 2.2e-16 = 4e-14, here 1e-13.  And a pattern that overflows:
it reaches the boxes that have it in their list 2 and no sibling of theirs."""
import os
import re

import numpy as np
import pytest

from mlfma_b200 import MLFMA, inputs

pytestmark = pytest.mark.gpu
PW = inputs.PlaneWave()
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlfma_b200", "csrc")


def min_pair_dirs():
    with open(os.path.join(CSRC, "device.cuh")) as f:
        return int(re.search(r"kM2LMinPairDirs = (\d+);", f.read()).group(1))


def lists(op):
    """Per level and parent: the list-2 lengths of its boxes that hold sources."""
    nodes, l2 = op.tree_export(0).reshape(-1, 14), op.tree_export(4)
    out, at = {}, 0
    for level, parent, count in nodes[:, [0, 1, 13]]:
        if count > 0:
            out.setdefault(int(level), {}).setdefault(int(parent), []).append(int(l2[at]))
        at += 1 + int(l2[at])
    return out


def family_levels(op):
    found = {}
    for level, sib in lists(op).items():
        if level < 2:
            continue
        g = op.level_info(level)
        if sum(map(sum, sib.values())) * g["nth"] * g["nph"] >= min_pair_dirs():
            found[level] = sib
    return found


def scattered(seed):
    """A dense half of the root box and, well apart from it, two small clusters (one
    of a single leaf, one of several), a thin one along the half's far edge and a few
    sources in corners."""
    r = np.random.default_rng(seed)
    dense = r.uniform([-1.99, -1.99, -1.99], [-0.01, 1.99, 1.99], (6000, 3))
    one = r.uniform([1.51, 1.51, 1.51], [1.74, 1.74, 1.74], (4, 3))
    many = r.uniform([1.01, -1.99, -1.99], [1.99, -1.01, -1.01], (300, 3))
    thin = r.uniform([0.01, -0.1, 0.3], [0.49, 0.1, 0.4], (40, 3))
    pos = np.concatenate([dense, one, many, thin])
    return inputs.Dipoles(pos=pos, mom=np.tile([0.0, 0.6, 0.8], (len(pos), 1)))


def cvec(n, seed):
    r = np.random.default_rng(seed)
    return r.standard_normal(n) + 1j * r.standard_normal(n)


@pytest.mark.parametrize("ref_compat", [0, 1])
@pytest.mark.parametrize("leaf,max_level,sizes", [(16, 4, {1, 2, 5, 6, 7, 8}), (2, 4, {1, 2, 5, 6, 7, 8}), (40, 3, {8})])
def test_families_with_empty_lists(cuda_device, leaf, max_level, sizes, ref_compat):
    ys = {}
    for sched in (0, 1):
        op = MLFMA.dipoles(scattered(7), PW, ref_compat=ref_compat, max_node_srcs=leaf, max_level=max_level).setup()
        fam = family_levels(op)
        assert fam
        lens = [n for sib in fam.values() for group in sib.values() for n in group]
        groups = [group for sib in fam.values() for group in sib.values()]
        assert 0 in lens and max(lens) > 32                       # empty lists, more than one staged batch
        assert any(not any(g) for g in groups)                    # a family with nothing to translate
        assert sizes <= {len(g) for g in groups}                  # single boxes to all eight siblings
        op.set_schedule(sched)
        ys[sched] = [op.matvec(cvec(op.n, s)) for s in (1, 2, 3)]
        if not ref_compat:
            ys[sched].append(op.matvec_adjoint(cvec(op.n, 4)))
        op.close()
    for a, b in zip(ys[1], ys[0]):
        assert np.linalg.norm(a - b) <= 1e-13 * np.linalg.norm(b)


def test_overflow_reaches_only_its_list(cuda_device):
    # the sources of one leaf lie in a plane, along x, at 1.7e308: their pattern
    # overflows.  Sources in that plane along z, in the leaves around, have nothing
    # to do with them directly (entries of zero) nor through a list 2.
    d = inputs.make_dipoles(8192, seed=1)
    at = np.floor((d.pos + 2.0) / 0.5)
    cell = np.all(at == [3, 3, 3], axis=1)
    around = np.all(np.abs(at - 3) <= 1, axis=1) & ~cell
    plane = around & (at[:, 2] == 3)
    assert cell.sum() > 4 and plane.sum() > 40
    pos, mom = d.pos.copy(), np.tile([0.6, 0.0, 0.8], (d.n, 1))
    pos[cell | plane, 2] = -0.25
    mom[cell], mom[plane] = [1.0, 0.0, 0.0], [0.0, 0.0, 1.0]
    x = cvec(d.n, 5)
    x[cell] = 1.7e308
    for sched in (0, 1):
        op = MLFMA.dipoles(inputs.Dipoles(pos=pos, mom=mom), PW, ref_compat=0, max_node_srcs=64).setup()
        assert 3 in family_levels(op) and op.stats()["max_level"] == 3
        op.set_schedule(sched)
        finite = np.isfinite(op.matvec(x))
        assert not finite[~around & ~cell].any()
        assert finite[plane].all(), sched
        op.close()
