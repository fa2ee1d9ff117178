"""Set-up on the device: the PEC edge mask kernel against the host's, the field
layout round trip, and staged host <-> device copies of sizes around the staging
threshold and its slots."""

import numpy as np
import pytest
import torch

import oracle
from rfx_b200 import engine
from rfx_b200.engine import Plan, PlanSpec, to_host

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


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 5, 31), (9, 2, 128), (4, 7, 129), (2, 33, 300), (120, 90, 33)])
def test_fields_round_trip_through_the_padded_layout(cuda, shape):
    p = _plan(shape)
    try:
        f = np.random.default_rng(3).standard_normal((6,) + shape).astype(np.float32)
        p.load_fields(list(f))
        for a, b in zip(f, p.store_fields()):
            assert np.array_equal(a, b.cpu().numpy())
    finally:
        p.close()


@pytest.mark.parametrize("extra", [-1, 0, 1, engine._STAGE_BYTES // 4 + 3, 3 * engine._STAGE_BYTES // 4 - 1])
def test_staged_copies_round_trip(cuda, extra):
    p = _plan((4, 4, 4))
    try:
        n = engine._STAGED_UP // 4 + extra
        a = np.random.default_rng(2).standard_normal(n).astype(np.float32)
        d = p._dev(a)
        assert np.array_equal(d.cpu().numpy(), a)
        x, y = to_host([d, d * 2.0])
        assert np.array_equal(x, a) and np.array_equal(y, a * np.float32(2.0))
        assert x.flags.writeable and x.base is not y.base
    finally:
        p.close()
