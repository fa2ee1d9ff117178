"""A reverse pass repeated on the same forward history gives the same bits, and so
does the pass over recomputed segments: every adjoint value has one writer per
step and a fixed order of operations.  Several hundred steps of a grid whose every
tile lies in a slab, and of one with CPML-free items, so that a value read before
it is written, or after its place is taken again, would show."""

import numpy as np
import pytest
import torch

from rfx_b200 import MaterialArrays, workloads
from rfx_b200.adjoint import AdjointRunner
from rfx_b200.grid import Grid


def _scene(kind, n):
    if kind == "slabs everywhere":
        g, eps, sig, src, probes, box, _ = workloads.adjoint_region(n_steps=n)
        return g, eps, sig, src, probes, box
    shape = (180, 107, 109)
    g = Grid(freq_max=20e9, domain=tuple((s - 17) * 1e-3 for s in shape), dx=1e-3, cpml_layers=8)
    assert g.shape == shape
    rng = np.random.default_rng(2)
    eps = (1.0 + rng.random(shape)).astype(np.float32)
    src = [(90, 50, 54, "ez", rng.standard_normal(n).astype(np.float32))]
    probes = [(90 + 2 * q, 54, 52 + q, c) for q, c in enumerate(("ez", "hy", "ex"))]
    return g, eps, np.zeros(shape, np.float32), src, probes, (80, 100, 40, 60, 45, 60)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["slabs everywhere", "CPML-free items"])
def test_repeated_reverse_passes_agree_bit_for_bit(cuda, kind):
    n = 600
    g, eps, sig, src, probes, box = _scene(kind, n)
    mats = MaterialArrays(eps, sig, np.ones_like(eps))
    kw = dict(sources=src, probes=probes, box=box, boundary="cpml", cpml_axes="xyz", pec_axes="")
    a = AdjointRunner(g, mats, n, mode="history", **kw)
    b = AdjointRunner(g, mats, n, mode="segments", checkpoint_every=64, **kw)
    try:
        ts = a.forward().clone()
        gvec = torch.from_numpy(np.random.default_rng(5).standard_normal(tuple(ts.shape)).astype(np.float32)).cuda()
        grad, src_adj = (t.clone() for t in a.backward(gvec))
        assert float(grad.abs().max()) > 0 and float(src_adj.abs().max()) > 0
        for _ in range(4):
            again = a.backward(gvec)
            assert torch.equal(again[0], grad) and torch.equal(again[1], src_adj)
        assert torch.equal(b.forward(), ts)
        again = b.backward(gvec)
        assert torch.equal(again[0], grad) and torch.equal(again[1], src_adj)
    finally:
        a.close()
        b.close()
