"""Rounding of the forward step's CPML terms.

Grids with an 8 x 32 tile that reaches both slabs of an axis, or with more than 16
layers, take a psi term from g = difference * (1 / cell) and the profile's own b, c
and 1/kappa - 1, as the kernel with one cell per thread (RFXB_STAGING=cpasync)
does; without kappa grading the results are its results bit for bit, from the
kernels with four cells per thread and the one-launch advance alike.  (With 1 / cell
divided into c, every c is rounded once more and the fields were up to 1.13 times
as far from a float64 march.)  Other grids take the divided coefficients.

kappa_max > 1 adds the curl's own term: forward and reverse step against the
float64 oracle.  Per step a cell takes some twenty roundings of 2^-24, which add
up like a random walk: 6e-8 sqrt(20 n) for n steps, 2e-6 for 60 steps, of which
four times are the limit here.
"""

import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
from oracle.adjoint import forward_adjoint
from rfx_b200.grid import Grid
from rfx_b200.simulation import MaterialArrays, prepare_device_run
from tests.test_gpu_fullsize import COMPONENTS, _advance, _random_fields

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# cells, CPML layers, CPML axes, per-cell mu_r
SCENES = [((43, 37, 33), 6, "xyz", False), ((36, 52, 39), 8, "xyz", False), ((60, 33, 36), 6, "yz", True),
          ((47, 22, 70), 8, "y", False), ((50, 30, 21), 5, "z", True), ((60, 45, 77), 18, "xyz", False),
          ((80, 200, 38), 7, "xz", False)]
OTHER = ((64, 52, 49), 8, "xyz", False)   # divided coefficients
STEPS = 24


def _grid(shape, ncp, kappa_max=1.0):
    g = Grid(freq_max=20e9, domain=tuple((n - 2 * ncp - 1) * 1e-3 for n in shape), dx=1e-3, cpml_layers=ncp,
             kappa_max=kappa_max)
    assert g.shape == shape
    return g


def _run(scene, n=STEPS, kappa_max=1.0):
    """Device run of a scene, with its seed fields, materials and source."""
    shape, ncp, axes, mu_cells = scene
    rng = np.random.default_rng(sum(shape))
    eps = (1.0 + 3.0 * rng.random(shape)).astype(np.float32)
    sig = (0.02 * rng.random(shape)).astype(np.float32)
    mu = (1.0 + rng.random(shape)).astype(np.float32) if mu_cells else np.ones(shape, np.float32)
    c = tuple(s // 2 for s in shape)
    src = [(*c, "ez", rng.standard_normal(n).astype(np.float32))]
    r = prepare_device_run(_grid(shape, ncp, kappa_max), MaterialArrays(eps, sig, mu), n, cpml_axes=axes, pec_axes="",
                           sources=src, probes=[(c[0] + 2, c[1], c[2], "hy")], dft_planes=[], pec_mask=None,
                           dft_time_offset=1)
    return r, _random_fields(shape, 5), (eps, sig, mu), src


def _march(r, init, n, chunks):
    _, _ = _advance(r, n, init=init, chunks=chunks)
    return [f.cpu().numpy().copy() for f in r.plan.store_fields()]


def _main(path):
    out = {}
    for q, scene in enumerate(SCENES + [OTHER]):
        r, init, _, _ = _run(scene)
        for c, f in zip(COMPONENTS, _march(r, init, STEPS, 1)):
            out[f"{c}{q}"] = f
        assert r.plan.forward_variant() == 0
        r.plan.close()
    np.savez(path, **out)


@pytest.mark.gpu
def test_forward_step_rounds_as_one_cell_per_thread(cuda, tmp_path):
    path = str(tmp_path / "one_cell.npz")
    env = dict(os.environ, RFXB_STAGING="cpasync", PYTHONPATH=ROOT)
    code = f"from tests.test_gpu_forward_rounding import _main; _main({path!r})"
    p = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    one = np.load(path)
    for q, scene in enumerate(SCENES + [OTHER]):
        r, init, _, _ = _run(scene)
        try:
            assert r.plan.forward_variant() == 2
            for chunks, route in ((1, 1 if scene[3] else 2), (STEPS, 1)):
                got = _march(r, init, STEPS, chunks)
                assert np.prod(scene[0]) > 606208 or r.plan.forward_route()[0] == route
                for c, f in zip(COMPONENTS, got):
                    if scene is OTHER:
                        assert np.linalg.norm(f - one[f"{c}{q}"]) < 2e-6 * np.linalg.norm(f)
                    else:
                        assert np.array_equal(f, one[f"{c}{q}"]), (scene, chunks, c)
        finally:
            r.plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("scene", SCENES[:3] + [OTHER])
def test_forward_with_kappa_grading_matches_float64(cuda, scene):
    n, kappa = 60, 5.0
    r, init, mats, src = _run(scene, n, kappa)
    shape, ncp, axes, _ = scene
    og = oracle.make_uniform_grid(tuple((s - 2 * ncp - 1) * 1e-3 for s in shape), 1e-3, cpml_layers=ncp)
    assert tuple(og.shape) == shape
    ref, flat = (oracle.run_uniform(og, mats, n, cpml_axes=axes, pec_axes="", sources=src, dtype=np.float64,
                                    kappa_max=k, init_fields=init).state for k in (kappa, 1.0))
    try:
        for chunks, route in ((1, 1 if scene[3] else 2), (n, 1)):
            got = _march(r, init, n, chunks)
            assert r.plan.forward_route()[0] == route
            for c, f in zip(COMPONENTS, got):
                e = np.linalg.norm(f - ref[c]) / np.linalg.norm(ref[c])
                print(scene, chunks, c, "error against float64", e)
                assert e < 8e-6
                assert np.linalg.norm(flat[c] - ref[c]) > 1e-3 * np.linalg.norm(ref[c])   # kappa counts
    finally:
        r.plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("shape,ncp,axes", [((300, 41, 97), 8, "xyz"), ((400, 47, 73), 4, "yz")])
def test_tile_shapes_agree_with_kappa_grading(cuda, shape, ncp, axes):
    r, init, _, _ = _run((shape, ncp, axes, False), 7, 5.0)
    try:
        r.plan.set_launch_config(fwd_split=0)
        single = _march(r, init, 7, 1)
        assert r.plan.forward_route() == (1, 24)
        r.plan.set_launch_config(fwd_split=1)
        for a, b in zip(single, _march(r, init, 7, 1)):
            assert np.array_equal(a, b)
    finally:
        r.plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("inner,ncp,mu_cells", [((24, 26, 20), 6, False), ((30, 18, 16), 5, True)])
def test_reverse_with_kappa_grading_matches_float64(cuda, inner, ncp, mu_cells):
    import torch

    import rfx_b200
    from rfx_b200.adjoint import AdjointRunner
    n, kappa, dx = 60, 5.0, 1e-3
    rng = np.random.default_rng(ncp)
    domain = tuple((v - 0.5) * dx for v in inner)
    og = oracle.make_uniform_grid(domain, dx, cpml_layers=ncp)
    shape = tuple(og.shape)
    eps = (1.0 + 2.0 * rng.random(shape)).astype(np.float32)
    sig = (0.02 * rng.random(shape)).astype(np.float32)
    mu = (1.0 + rng.random(shape)).astype(np.float32) if mu_cells else np.ones(shape, np.float32)
    # sources and probes in the slabs too: the gradient passes through them
    cell = lambda m: tuple(int(rng.integers(m, s - m)) for s in shape)   # noqa: E731
    sources = [(*cell(1), COMPONENTS[q % 3], rng.standard_normal(n).astype(np.float32)) for q in range(40)]
    probes = [(*cell(1), COMPONENTS[q % 6]) for q in range(36)]
    cot = (rng.standard_normal((n, 36)) * [1.0 if q % 6 < 3 else 377.0 for q in range(36)]).astype(np.float32)
    a = ncp + 3
    box = (a, a + 6, a, a + 5, a, a + 4)
    kw = dict(boundary="cpml", pec_axes="", sources=sources, probes=probes, box=box,
              objective_grad=lambda ts: cot.astype(np.float64))
    _, g64, s64 = forward_adjoint(og, (eps, sig, mu), n, kappa_max=kappa, **kw)
    _, _, flat = forward_adjoint(og, (eps, sig, mu), n, **kw)
    g = rfx_b200.Grid(freq_max=10e9, domain=domain, dx=dx, cpml_layers=ncp, kappa_max=kappa)
    assert tuple(g.shape) == shape
    r = AdjointRunner(g, rfx_b200.MaterialArrays(eps, sig, mu), n, sources=sources, probes=probes, box=box,
                      boundary="cpml", cpml_axes="xyz", pec_axes="")
    try:
        r.forward()
        grad, src = (t.cpu().numpy() for t in r.backward(torch.from_numpy(cot).cuda()))
        assert r.plan.adjoint_variant() == 2
    finally:
        r.close()
    es, eg = np.linalg.norm(src - s64) / np.linalg.norm(s64), np.linalg.norm(grad - g64) / np.linalg.norm(g64)
    print("source adjoint", es, "gradient", eg)
    assert es < 8e-6 and eg < 8e-6
    assert np.linalg.norm(flat - s64) > 1e-3 * np.linalg.norm(s64)
