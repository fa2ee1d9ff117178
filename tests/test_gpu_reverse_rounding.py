"""Rounding of the four-cells-per-thread reverse step against the kernel with one
cell per thread (RFXB_STAGING=cpasync), whose differences of products have one
product rounded and the other fused.

The adjoint of the source table samples the adjoint E at many cells after every
step and does not depend on the forward march, so against the float64 oracle it
shows the rounding of the reverse step alone.  Without CPML both kernels do the
same operations and agree bit for bit.  In the slabs the flux of a cell and its
relation are added in another order: as many roundings, so the errors agree up to
the sampling of 240 cells (0.97 to 1.02 a scene, 0.996 over them).  With every
product of a flux rounded the error was 1.04 to 1.17 times the other kernel's.

The scenes have more sources and probes than one mask word holds, E and H probes,
lossy boxes and, in one, per-cell mu_r.
"""

import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
from oracle.adjoint import forward_adjoint

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
COMPS = ("ex", "ey", "ez", "hx", "hy", "hz")
STEPS = 120
# cells between the slabs, CPML layers, per-cell mu_r
SCENES = [((40, 36, 44), 6, False), ((44, 50, 40), 8, False), ((30, 60, 44), 6, False), ((40, 36, 44), 6, True),
          ((50, 34, 50), 0, False)]


def _scene(q):
    inner, ncp, mu_cells = SCENES[q]
    rng = np.random.default_rng(q)
    dx = 1e-3
    domain = tuple((n - 0.5) * dx for n in inner)
    g = oracle.make_uniform_grid(domain, dx, cpml_layers=ncp)
    eps, sig, mu = (np.ones(g.shape, np.float32) for _ in range(3))
    sig[:] = 0.0
    for _ in range(5):
        lo, size = [int(rng.integers(0, n - 8)) for n in g.shape], rng.integers(4, 20, 3)
        sl = tuple(slice(a, a + b) for a, b in zip(lo, size))
        eps[sl], sig[sl] = rng.uniform(1, 5), rng.uniform(0, 0.05)
    if mu_cells:
        mu[: g.shape[0] // 2] = 2.2
    t = np.arange(STEPS) * g.dt

    def wave():   # a carrier ramped up over a period
        f = rng.uniform(6e9, 12e9)
        return (np.sin(2 * np.pi * f * t + rng.uniform(0, 6)) * (1 - np.exp(-(t * f) ** 2))).astype(np.float32)

    def cell(m):
        return tuple(int(rng.integers(m, n - m)) for n in g.shape)

    sources = [(*cell(1), COMPS[p % 3], wave()) for p in range(240)]
    probes = [(*cell(ncp + 2), COMPS[p % 6]) for p in range(48)]
    cot = np.stack([wave()[::-1] * (1.0 if p % 6 < 3 else 377.0) for p in range(48)], 1).astype(np.float32)
    a = ncp + 4
    return g, domain, (eps, sig, mu), sources, probes, cot, (a, a + 5, a, a + 5, a + 1, a + 4), ncp


def _reverse(q):
    import torch

    import rfx_b200
    from rfx_b200.adjoint import AdjointRunner
    og, domain, mats, sources, probes, cot, box, ncp = _scene(q)
    g = rfx_b200.Grid(freq_max=10e9, domain=domain, dx=og.dx, cpml_layers=ncp)
    assert tuple(g.shape) == tuple(og.shape)
    r = AdjointRunner(g, rfx_b200.MaterialArrays(*mats), STEPS, sources=sources, probes=probes, box=box,
                      boundary="cpml" if ncp else "pec", cpml_axes="xyz" if ncp else "", pec_axes="" if ncp else "xyz")
    try:
        r.forward()
        grad, src = r.backward(torch.from_numpy(cot).cuda())
        return grad.cpu().numpy(), src.cpu().numpy(), r.plan.adjoint_variant()
    finally:
        r.close()


def _main(path):
    out = {}
    for q in range(len(SCENES)):
        grad, src, variant = _reverse(q)
        assert variant == 0
        out[f"grad{q}"], out[f"src{q}"] = grad, src
    np.savez(path, **out)


@pytest.mark.gpu
def test_reverse_step_rounds_as_well_as_one_cell_per_thread(cuda, tmp_path):
    path = str(tmp_path / "one_cell.npz")
    env = dict(os.environ, RFXB_STAGING="cpasync", PYTHONPATH=ROOT)
    code = f"from tests.test_gpu_reverse_rounding import _main; _main({path!r})"
    p = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    one = np.load(path)
    ratios = []
    for q, (_, ncp, _) in enumerate(SCENES):
        grad, src, variant = _reverse(q)
        assert variant == (2 if ncp else 3)
        if not ncp:
            assert np.array_equal(src, one[f"src{q}"]) and np.array_equal(grad, one[f"grad{q}"])
            continue
        og, _, mats, sources, probes, cot, box, _ = _scene(q)
        _, g64, s64 = forward_adjoint(og, mats, STEPS, boundary="cpml", pec_axes="", sources=sources, probes=probes,
                                      box=box, objective_grad=lambda ts: cot.astype(np.float64))
        err, err1 = (np.linalg.norm(a.astype(np.float64) - s64) / np.linalg.norm(s64) for a in (src, one[f"src{q}"]))
        print(SCENES[q], "error against float64", err, "one cell per thread", err1, "ratio", err / err1)
        assert err < 5e-6 and np.linalg.norm(grad - g64) < 2e-6 * np.linalg.norm(g64)
        ratios.append(err / err1)
    assert np.exp(np.mean(np.log(ratios))) < 1.04, ratios
