"""Products on host buffers: ordinary memory goes through the handle's own
page-locked buffer, page-locked memory through the driver's copies.  Both feed
the same kernels with the same values, so the results are equal bit for bit."""
import numpy as np
import pytest
import torch

from mlfma_b200 import MLFMA, inputs

pytestmark = pytest.mark.gpu


def locked(v):
    return torch.from_numpy(v.copy()).pin_memory().numpy()


@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("n", [2, 255, 257, 3000])
def test_both_routes_agree(cuda_device, n, accumulate):
    r = np.random.default_rng(n)
    op = MLFMA.dipoles(inputs.make_dipoles(n, seed=n), inputs.PlaneWave(), max_node_srcs=24, ref_compat=0).setup()
    x, y, z = (r.standard_normal(n) + 1j * r.standard_normal(n) for _ in range(3))
    op.set_loads(z)
    for product in (op.matvec, op.matvec_adjoint):
        a = product(x, accumulate=accumulate, out=y.copy())
        b = product(locked(x), accumulate=accumulate, out=locked(y))
        assert np.array_equal(a, b)
        assert not np.array_equal(a, y)
    op.close()
