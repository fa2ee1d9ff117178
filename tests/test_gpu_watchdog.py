"""Device-side failure paths of the step kernels, exercised without faulting
the GPU: a pipeline wait made to run out (one CTA does not issue one plane's
TMA boxes, every wait is limited to some polls), a grid barrier whose wait is
limited to one poll, and a poisoned work-queue entry (an empty x range) of the
persistent kernels.  In every case the kernels finish, the status word reports the failure to the host
(RFXB_E_TIMEOUT = -6, RFXB_E_WORK = -7), and a fresh sweep on the same
device afterwards runs clean and reproduces the undisturbed result bit for
bit."""

import numpy as np
import pytest


def _sweep():
    import torch

    from rfx_b200.batch import Sweep
    from rfx_b200.workloads import batched_sweep
    insts = batched_sweep(seed=3, n_inst=3, n_steps=60, n_lo=40, n_hi=72)
    sw = Sweep(insts, 60, device=torch.device("cuda", 0), batched=True)
    _, lim = sw.batch.launch_config()
    assert lim["fwd_persist"] >= 1 and lim["adj_persist"] == 1
    sw.batch.set_launch_config(fwd_persist=2, adj_persist=1)
    return sw


def _result(sw):
    Js, grads = sw.run()
    sw.check_device()
    return np.array([float(j) for j in Js]), [g.detach().cpu().numpy().copy() for g in grads]


def _lib():
    from rfx_b200 import _lib
    return _lib.load()


def _clean_rerun_matches(J0, g0):
    sw = _sweep()
    try:
        J, g = _result(sw)
        assert np.array_equal(J, J0)
        for a, b in zip(g, g0):
            assert np.array_equal(a, b)
    finally:
        sw.close()


@pytest.mark.gpu
def test_forward_wait_that_runs_out_is_reported(cuda):
    sw = _sweep()
    try:
        J0, g0 = _result(sw)
        assert _lib().rfxb_batch_debug_fault(sw.batch._h, 0, 256) == 0
        sw.forward()
        with pytest.raises(RuntimeError, match=r"code -6\).*ran out"):
            sw.check_device()
    finally:
        sw.close()
    _clean_rerun_matches(J0, g0)


@pytest.mark.gpu
def test_reverse_wait_that_runs_out_is_reported(cuda):
    sw = _sweep()
    try:
        J0, g0 = _result(sw)
        sw.forward()
        _, gs = sw.objectives()
        sw.check_device()
        assert _lib().rfxb_batch_debug_fault(sw.batch._h, 0, 256) == 0
        sw.backward(gs)
        with pytest.raises(RuntimeError, match=r"code -6\).*ran out"):
            sw.check_device()
    finally:
        sw.close()
    _clean_rerun_matches(J0, g0)


@pytest.mark.gpu
@pytest.mark.parametrize("which", [0, 1, 4])
def test_poisoned_work_item_is_rejected(cuda, which):
    """Lists 0 / 1: forward CPML / CPML-free tiles; 4: reverse CPML-free."""
    sw = _sweep()
    try:
        J0, g0 = _result(sw)
        assert _lib().rfxb_batch_debug_poison(sw.batch._h, which, 0) == 0
        if which < 2:
            sw.forward()
        else:
            sw.forward()
            _, gs = sw.objectives()
            sw.backward(gs)
        with pytest.raises(RuntimeError, match=r"code -7\).*invalid work item"):
            sw.check_device()
    finally:
        sw.close()
    _clean_rerun_matches(J0, g0)


def _device_runs(shapes, ncp, n):
    from rfx_b200.grid import Grid
    from rfx_b200.simulation import MaterialArrays, prepare_device_run
    runs = []
    for shape in shapes:
        rng = np.random.default_rng(shape[0])
        g = Grid(freq_max=20e9, domain=tuple((s - 2 * ncp - 1) * 1e-3 for s in shape), dx=1e-3, cpml_layers=ncp)
        assert g.shape == shape
        eps = (1.0 + rng.random(shape)).astype(np.float32)
        c = tuple(s // 2 for s in shape)
        runs.append(prepare_device_run(
            g, MaterialArrays(eps, np.zeros(shape, np.float32), np.ones(shape, np.float32)), n,
            cpml_axes="xyz" if ncp else "", pec_axes="" if ncp else "xyz",
            sources=[(*c, "ez", rng.standard_normal(n).astype(np.float32))], probes=[(c[0] + 2, c[1], c[2], "ez")],
            dft_planes=[], pec_mask=None, dft_time_offset=1))
    return runs


# grids, CPML layers, launch fields, (route, tile rows), block whose wait runs out, poll limit
FORWARD = {
    "two-step passes, faces": ([(64, 80, 96)], 0, dict(fwd_depth=2), (1, 8), 0, 1 << 14),
    "two-step passes, interior": ([(64, 80, 128)], 8, dict(fwd_depth=2), (1, 8), 1, 1 << 14),
    "one launch for all steps": ([(61, 52, 49)], 8, {}, (2, 8), -1, 1),
}


@pytest.mark.gpu
@pytest.mark.parametrize("kind", list(FORWARD))
def test_forward_wait_off_the_queues_that_runs_out_is_reported(cuda, kind):
    import torch

    from rfx_b200.engine import Batch
    shapes, ncp, config, route, cta, limit = FORWARD[kind]
    n = 6

    def march(fault):
        runs = _device_runs(shapes, ncp, n)
        b = Batch([r.plan for r in runs])
        try:
            if config:
                b.set_launch_config(**config)
            if fault:
                assert _lib().rfxb_batch_debug_fault(b._h, cta, limit) == 0
            b.advance(0, n, [dict(src_table=r.src_table, probe_out=r.probe_out) for r in runs])
            torch.cuda.synchronize()
            assert b.forward_route() == route
            if fault:
                with pytest.raises(RuntimeError, match=r"code -6\).*ran out"):
                    b.check_device()
                return None
            b.check_device()
            return [f.cpu().numpy().copy() for r in runs for f in r.plan.store_fields()]
        finally:
            b.close()
            for r in runs:
                r.plan.close()

    ref = march(False)
    march(True)
    for x, y in zip(ref, march(False)):
        assert np.abs(x).max() > 0 and np.array_equal(x, y)
