"""The subgrid transforms of the device calls (register form) at every subgrid size, w-stacked and not, odd
grids and negative w, against the host-array calls of the same plan, which run the other form.

Either is within 1e-6 of the FP64 result in FP32 mode (their stated bar is 1e-5), so they differ by at
most 2e-6.
"""
import numpy as np
import pytest

from conftest import constants, pkg, rel_l2, workload

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TOL = 2e-6


@pytest.mark.parametrize("S,kernel", [(8, 2), (16, 4), (24, 8), (32, 8), (48, 8)])
@pytest.mark.parametrize("N", [256, 257])
@pytest.mark.parametrize("wstack", [True, False])
def test_device_matches_host(need_gpu, S, kernel, N, wstack):
    obs, cd = workload("small_256", n_ant=7, nt=90, nch=3, seed=S)
    c, cd = constants(cd, grid_size=N, subgrid_size=S, kernel_size=kernel, wstep=cd["wstep"] * (1 + 1e-6))
    part = pkg.Partitioner.CreatePartition(c, obs.uvw, obs.frequencies)
    plan, W = part.plan, cd["wlayer_count"] if wstack else 1
    vis = obs.vis.astype(np.complex64)
    d_vis = torch.from_numpy(vis).cuda()
    d_grid = torch.full((W, N, N), float("nan"), dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    (plan.grid_w_device if wstack else plan.grid_device)(d_vis.data_ptr(), d_grid.data_ptr())
    plan.synchronize()
    host = (pkg.IDG.GridW if wstack else pkg.IDG.Grid)(c, part, vis.astype(np.complex128), obs.uvw, obs.frequencies)
    assert rel_l2(d_grid.cpu().numpy().reshape(host.shape), host) < TOL
    rng = np.random.default_rng(S + N)
    model = (rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))).astype(np.complex64)
    d_model = torch.from_numpy(model).cuda()
    d_out = torch.full(vis.shape, float("nan"), dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    (plan.degrid_w_device if wstack else plan.degrid_device)(d_model.data_ptr(), d_out.data_ptr())
    plan.synchronize()
    degrid = pkg.IDG.DeGridW if wstack else pkg.IDG.DeGrid
    host = degrid(c, part, model.astype(np.complex128), obs.uvw, obs.frequencies)
    assert rel_l2(d_out.cpu().numpy(), host) < TOL
