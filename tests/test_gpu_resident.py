"""An advance of a small grid runs in one launch that keeps the state in shared
memory; it gives the results of one launch per step, bit for bit.

Advances of one step each take the step kernels, so the two are compared on
grids whose blocks end on, before and after the grid's faces, from a few cells
to the largest that fits, axes so thin that tiles reach both slabs, CPML on some axes,
odd and even step counts, chunks, graded spacing, a PEC sheet, and more sources
and probes than one mask word holds.
"""

import numpy as np
import pytest
import torch

from rfx_b200 import _lib, workloads
from rfx_b200.engine import Batch
from rfx_b200.grid import Grid, make_nonuniform_grid
from rfx_b200.simulation import MaterialArrays, prepare_device_run
from tests.test_gpu_fullsize import _advance, _random_fields

pytestmark = pytest.mark.gpu

CASES = [((87, 47, 42), 8, "xyz", "", 1), ((33, 29, 31), 6, "yz", "x", 40), ((5, 4, 3), 0, "", "xyz", 1),
         ((61, 1 + 52, 49), 8, "x", "yz", 3), ((97, 77, 75), 0, "", "xyz", 2), ((40, 21, 150), 5, "xyz", "", 2), ((24, 22, 20), 4, "xyz", "", 2),
         ((2, 2, 2), 0, "", "xyz", 1), ((19, 31, 11), 3, "xz", "y", 3)]


def _compare(r, shape, n):
    init = _random_fields(shape, 7)
    runs = []
    for chunks in (n, 1, 3):
        ts, _ = _advance(r, n, init=init, chunks=chunks)
        assert r.plan.forward_route()[0] == (1 if chunks == n else 2)
        runs.append([ts] + [f.cpu().numpy().copy() for f in r.plan.store_fields()] +
                    [r.plan.save_state()])
    for other in runs[1:]:
        for a, b in zip(runs[0], other):
            assert np.array_equal(a, b)
    assert np.abs(runs[0][1]).max() > 0


@pytest.mark.parametrize("shape,ncp,cpml_axes,pec_axes,points", CASES)
@pytest.mark.parametrize("n", [6, 7])
def test_resident_advance_equals_steps(cuda, shape, ncp, cpml_axes, pec_axes, points, n):
    rng = np.random.default_rng(2)
    g = Grid(freq_max=20e9, domain=tuple((s - 2 * ncp - 1) * 1e-3 for s in shape), dx=1e-3, cpml_layers=ncp)
    assert g.shape == shape
    eps = (1.0 + rng.random(shape)).astype(np.float32)
    sig = (0.02 * rng.random(shape)).astype(np.float32)
    at = [tuple(int(rng.integers(0, s)) for s in shape) for _ in range(2 * points)]
    src = [(*c, ("ex", "ey", "ez")[q % 3], rng.standard_normal(n).astype(np.float32)) for q, c in enumerate(at[:points])]
    prb = [(*c, ("ez", "hx", "ey", "hz", "ex", "hy")[q % 6]) for q, c in enumerate(at[points:] + [at[0]])]
    pec = np.zeros(shape, bool)
    pec[1:-1, 1:-1, shape[2] // 2] = True
    r = prepare_device_run(g, MaterialArrays(eps, sig, np.ones(shape, np.float32)), n, cpml_axes=cpml_axes,
                           pec_axes=pec_axes, sources=src, probes=prb, dft_planes=[], pec_mask=pec, dft_time_offset=1)
    try:
        _compare(r, shape, n)
    finally:
        r.plan.close()


def test_resident_advance_on_graded_spacing(cuda):
    n, rng, dx = 9, np.random.default_rng(3), 0.5e-3
    g = make_nonuniform_grid((20 * dx, 16 * dx), workloads.graded_dz(3)[:22], dx, cpml_layers=6)
    eps = (1.0 + 3.0 * rng.random(g.shape)).astype(np.float32)
    c = tuple(s // 2 for s in g.shape)
    r = prepare_device_run(g, MaterialArrays(eps, np.zeros(g.shape, np.float32), np.ones(g.shape, np.float32)), n,
                           cpml_axes="xyz", pec_axes="xyz", sources=[(*c, "ez", rng.standard_normal(n).astype(np.float32))],
                           probes=[(c[0] + 2, c[1], c[2], "ez")], dft_planes=[], pec_mask=None, dft_time_offset=0)
    try:
        _compare(r, g.shape, n)
    finally:
        r.plan.close()


def _small_run(n, seed=4):
    shape, rng = (33, 29, 31), np.random.default_rng(seed)
    g = Grid(freq_max=20e9, domain=tuple((s - 13) * 1e-3 for s in shape), dx=1e-3, cpml_layers=6)
    eps = (1.0 + rng.random(shape)).astype(np.float32)
    return prepare_device_run(g, MaterialArrays(eps, np.zeros(shape, np.float32), np.ones(shape, np.float32)), n,
                              cpml_axes="xyz", pec_axes="",
                              sources=[(16, 14, 15, "ez", rng.standard_normal(n).astype(np.float32))],
                              probes=[(18, 14, 15, "ez")], dft_planes=[], pec_mask=None, dft_time_offset=1)


def _batch_advance(r, b, n):
    r.plan.reset()
    r.probe_out.zero_()
    b.advance(0, n, [dict(src_table=r.src_table, probe_out=r.probe_out)])
    torch.cuda.synchronize()
    b.check_device()
    return [r.probe_out.cpu().numpy().copy()] + [f.cpu().numpy().copy() for f in r.plan.store_fields()]


def test_refused_resident_launch_takes_step_launches(cuda):
    """A cooperative launch that the driver does not take (the launch is not made
    here, its error code is) leaves the advance to the step launches."""
    n = 12
    r = _small_run(n)
    b = Batch([r.plan])
    try:
        ref = _batch_advance(r, b, n)
        assert b.forward_route()[0] == 2 and np.abs(ref[0]).max() > 0
        assert _lib.load().rfxb_batch_debug_refuse_resident(b._h, 1) == 0
        for _ in range(2):
            got = _batch_advance(r, b, n)
            assert b.forward_route()[0] == 1
            for x, y in zip(ref, got):
                assert np.array_equal(x, y)
    finally:
        b.close()
        r.plan.close()
