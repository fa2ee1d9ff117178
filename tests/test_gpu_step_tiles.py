"""The four-cells-per-thread step kernels give one result, bit for bit, on every
tile shape and list they are launched with.

Each product and sum of the forward and reverse step is rounded explicitly, so
the single launch (24 x 32 tiles on these grids, CPML-free items beside CPML
ones), the split launches (8 x 32 tiles) and the persistent launches must agree
exactly.  The 8 x 32 kernels are held to the float64 oracle by the parity
tests; the grids here are long in x and end one row or column past, at, and
short of a tile, with the high z slab on and off a 16-byte boundary of its psi
rows, so that partial quads, partial tiles and both psi access forms are met.
"""

import numpy as np
import pytest
import torch

from rfx_b200.batch import Sweep, SweepInstance
from rfx_b200.grid import Grid
from rfx_b200.simulation import MaterialArrays, prepare_device_run
from tests.test_gpu_fullsize import _advance, _random_fields

pytestmark = pytest.mark.gpu

# cells, CPML layers, CPML axes
GRIDS = [((300, 41, 97), 8, "xyz"), ((400, 48, 80), 10, "xyz"), ((400, 47, 73), 4, "yz"), ((600, 24, 97), 5, "z"),
         ((600, 73, 30), 6, "x")]


def _grid(shape, ncp):
    g = Grid(freq_max=20e9, domain=tuple((n - 2 * ncp - 1) * 1e-3 for n in shape), dx=1e-3, cpml_layers=ncp)
    assert g.shape == shape
    return g


@pytest.mark.parametrize("shape,ncp,axes", GRIDS)
@pytest.mark.parametrize("mu", [False, True])
def test_forward_lists_agree_bit_for_bit(cuda, shape, ncp, axes, mu):
    g, n = _grid(shape, ncp), 7
    rng = np.random.default_rng(3)
    eps = (1.0 + 3.0 * rng.random(shape)).astype(np.float32)
    mu_r = (1.0 + rng.random(shape)).astype(np.float32) if mu else np.ones(shape, np.float32)
    c = tuple(s // 2 for s in shape)
    src = [(*c, "ez", rng.standard_normal(n).astype(np.float32)),
           (c[0] - 3, 1, shape[2] - 2, "ex", rng.standard_normal(n).astype(np.float32))]
    prb = [(c[0] + 5, c[1], c[2], comp) for comp in ("ex", "ey", "ez", "hx", "hy", "hz")]
    pec = np.zeros(shape, bool)
    pec[20:40, 3:20, c[2]] = True
    r = prepare_device_run(g, MaterialArrays(eps, np.zeros(shape, np.float32), mu_r), n, cpml_axes=axes,
                           pec_axes="" if axes == "xyz" else "xyz", sources=src, probes=prb, dft_planes=[],
                           pec_mask=pec, dft_time_offset=1)
    init = _random_fields(shape, 4)

    def run(**config):
        r.plan.set_launch_config(**config)
        ts, _ = _advance(r, n, init=init)
        return [ts] + [f.cpu().numpy().copy() for f in r.plan.store_fields()]

    try:
        lim = r.plan.launch_config()[1]
        single = run(fwd_split=0)
        assert r.plan.forward_route() == (1, 24)
        assert np.abs(single[0]).max() > 0
        others = ([dict(fwd_split=1)] if lim["fwd_split"] else []) + \
                 ([dict(fwd_split=0, fwd_persist=2)] if lim["fwd_persist"] else [])
        assert others
        for config in others:
            for a, b in zip(single, run(**config)):
                assert np.array_equal(a, b), config
    finally:
        r.plan.close()


@pytest.mark.parametrize("shape,ncp,axes", GRIDS)
def test_reverse_lists_agree_bit_for_bit(cuda, shape, ncp, axes):
    g, n = _grid(shape, ncp), 24
    rng = np.random.default_rng(5)
    eps = (1.0 + 3.0 * rng.random(shape)).astype(np.float32)
    c = tuple(s // 2 for s in shape)
    src = [(*c, "ez", rng.standard_normal(n).astype(np.float32))]
    prb = [(c[0] + 4, c[1] + 2, c[2], "ez"), (c[0] + 2, c[1], c[2] + 3, "hy")]
    box = (c[0] - 9, c[0] + 9, 2, shape[1] - 1, c[2] - 7, c[2] + 6)
    inst = SweepInstance(grid=g, eps_r=eps, sigma=np.zeros(shape, np.float32), sources=src, probes=prb, box=box,
                         freqs=np.array([9e9, 12e9]), cpml_axes=axes, pec_axes="" if axes == "xyz" else "xyz")
    sw = Sweep([inst], n, device=torch.device("cuda", 0), batched=True)

    def run(**config):
        sw.batch.set_launch_config(**config)
        J, grads = sw.run()
        sw.check_device()
        return float(J[0]), grads[0].detach().cpu().numpy().copy()

    try:
        lim = sw.batch.launch_config()[1]
        J0, g0 = run(adj_lite=0)
        assert sw.batch.forward_route() == (1, 24)
        assert np.abs(g0).max() > 0
        others = ([dict(adj_lite=1)] if lim["adj_lite"] else []) + \
                 ([dict(adj_lite=0, adj_persist=1)] if lim["adj_persist"] else [])
        assert others
        for config in others:
            J, gr = run(**config)
            assert J == J0 and np.array_equal(gr, g0), config
    finally:
        sw.close()
