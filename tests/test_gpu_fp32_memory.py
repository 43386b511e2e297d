"""FP32 device calls without memory for the tensor cores' coefficients run the sincos kernels.

The plan's other buffers are made first, by calls on the sincos kernels; then each allocation of the tensor-core
state (coefficients, tables, work items) is made to fail (p9idg_debug_fail_device_allocations).
"""
import numpy as np
import pytest

from conftest import constants, oracle, pkg, rel_l2, workload

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _arm(after):
    assert pkg._native.lib().p9idg_debug_fail_device_allocations(after) == 0


def _setup():
    obs, cd = workload("small_256", n_ant=7, nt=160, nch=6)
    c, cd = constants(cd)
    N = cd["grid_size"]
    rng = np.random.default_rng(3)
    grid = (rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))).astype(np.complex64)
    subs = oracle.partition(cd, obs.uvw, obs.frequencies)
    ref = oracle.idg_grid_w(cd, subs, obs.vis.astype(np.complex64).astype(np.complex128), obs.uvw, obs.frequencies)
    vref, _ = oracle.idg_degrid(cd, subs, grid.astype(np.complex128), obs.uvw, obs.frequencies, wstack=True)
    bufs = [torch.from_numpy(obs.vis.astype(np.complex64)).cuda(), torch.empty(ref.shape, dtype=torch.complex64, device="cuda"),
            torch.from_numpy(grid).cuda(), torch.empty(obs.vis.shape, dtype=torch.complex64, device="cuda")]
    return obs, c, bufs, ref, vref


def _batch(plan, bufs):
    return pkg.Batch([plan], *([b.data_ptr()] for b in bufs))


@pytest.mark.parametrize("k", range(5))
def test_falls_back_to_sincos(need_gpu, k):
    obs, c, bufs, ref, vref = _setup()
    vis, layers, grid, out = bufs
    part = pkg.Partitioner.CreatePartition(c, obs.uvw, obs.frequencies)
    plan = part.plan
    pkg.set_chunking(plan, 64, 64)  # more partial subgrids for the sincos kernels than the tensor cores take
    plan.set_tc_order(2)            # kept when the tensor-core state is given up

    def calls():
        layers.fill_(float("nan"))
        out.fill_(float("nan"))
        torch.cuda.synchronize()
        plan.grid_w_device(vis.data_ptr(), layers.data_ptr())
        plan.degrid_w_device(grid.data_ptr(), out.data_ptr())
        plan.synchronize()
        assert rel_l2(layers.cpu().numpy(), ref) < 1e-5
        assert rel_l2(out.cpu().numpy(), vref) < 1e-5
        return plan.info()["device_form"]

    plan.set_fp32_tensor_cores(False)
    assert calls() == pkg.FORM_SINCOS
    plan.set_fp32_tensor_cores(True)
    _arm(k)
    try:
        form = calls()
    finally:
        _arm(-1)
    assert form == (pkg.FORM_SINCOS if k < 3 else pkg.FORM_TENSOR_CORE)
    assert calls() == form  # the plan keeps the form it went over to, and a batch takes it
    batch = _batch(plan, bufs)
    layers.fill_(float("nan"))
    out.fill_(float("nan"))
    torch.cuda.synchronize()
    batch.run()
    batch.synchronize()
    assert rel_l2(layers.cpu().numpy(), ref) < 1e-5
    assert rel_l2(out.cpu().numpy(), vref) < 1e-5
    batch.destroy()
    plan.set_fp32_tensor_cores(True)
    assert calls() == pkg.FORM_TENSOR_CORE
    assert plan.set_mode(pkg.MODE_TC_BF16X3) == pkg.MODE_TC_BF16X3 and plan.info()["tc_order"] == 2
