"""Set-up on the device: the PEC edge mask kernel against the host's."""

import numpy as np
import pytest

import oracle
from rfx_b200.engine import Plan, PlanSpec

pytestmark = pytest.mark.gpu


def _bits(m):
    x, y, z = (np.asarray(a, np.uint8) for a in oracle.tangential_edge_masks(m))
    return (x | y << 1 | z << 2).astype(np.uint8)


def _plan(shape):
    return Plan(PlanSpec(shape=shape, dt=1e-12, tables=[np.ones(n, np.float32) for n in np.repeat(shape, 2)]))


@pytest.mark.parametrize("shape", [(2, 2, 2), (5, 3, 7), (33, 31, 65), (180, 161, 160)])
def test_edge_mask_kernel_equals_host(cuda, shape):
    p = _plan(shape)
    try:
        rng = np.random.default_rng(1)
        for fill in (0.1, 0.6, 1.0):
            m = rng.random(shape) < fill
            assert np.array_equal(p.edge_mask(m).cpu().numpy(), _bits(m))
        # a mask in another memory order
        assert np.array_equal(p.edge_mask(np.asfortranarray(m)).cpu().numpy(), _bits(m))
    finally:
        p.close()
