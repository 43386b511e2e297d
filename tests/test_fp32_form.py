"""Which kernels the FP32 mode's device calls run.

On the tensor cores where the subgrids' samples lie close enough to their centre in w, |dw - dw0| |r| <=
8e-4, and there is enough work per subgrid, S^2 v > 128 (v + 375) for v visibilities a subgrid; else, and
wherever a program asks for them, the sincos kernels.  The choice is made on the host, so its edges are
tested without a GPU; GPU tests check that the calls run what the plan says.
"""
import numpy as np
import pytest

from conftest import constants, pkg, rel_l2, synth, workload

MAX_DEV = 8e-4


def remainder_max(cd):
    """max |r| of the pixels' n - f(x) - f(y), its range centred on zero (64 bits)."""
    S = cd["subgrid_size"]
    img = np.float64(np.float32(cd["scale_arcsec"]) * np.float32(cd["grid_size"]))
    l = (np.arange(S) - S // 2 + 0.5) * img / S
    n = lambda t: t / (t + np.sqrt(1 - t))  # noqa: E731  (ComputeN, Gridder.cs:168-174)
    r = n(l[:, None] ** 2 + l[None, :] ** 2) - n(l ** 2)[:, None] - n(l ** 2)[None, :]
    return 0.5 * (r.max() - r.min())


def deviation(part, cd, uvw, frequencies):
    k = 2 * np.pi * frequencies / 299792458.0
    dev = 0.0
    for s in part.plan.subgrids():
        t0, nt = int(s["time_sample_start"]), int(s["time_sample_count"])
        w = uvw[int(s["baseline_idx"]), t0:t0 + nt, 2]
        dev = max(dev, np.abs(w[:, None] * k[None, :] - w.mean() * k.mean()).max())
    return dev * remainder_max(cd)


def near_the_limit(share):
    """A 256^2 observation of a wide field (0.15 rad) with its w scaled to `share` of the limit."""
    obs, cd = workload("small_256", n_ant=8, nt=300, nch=8)
    uvw = obs.uvw.copy()
    uvw[..., :2] *= 0.05

    def plan(u):
        c, d = constants(cd, scale_arcsec=float(np.float32(0.15 / cd["grid_size"])),
                         wstep=synth.wstep_for(u, obs.frequencies, 4) * (1 + 1e-6), wlayer_count=4)
        return pkg.Partitioner.CreatePartition(c, u, obs.frequencies), c, d

    part, c, d = plan(uvw)
    uvw[..., 2] *= share * MAX_DEV / deviation(part, d, uvw, obs.frequencies)
    part, c, d = plan(uvw)
    assert deviation(part, d, uvw, obs.frequencies) == pytest.approx(share * MAX_DEV, rel=1e-3)
    return obs, uvw, part, c, d


@pytest.mark.parametrize("share,form", [(0.5, 1), (0.98, 1), (1.02, 0), (3.0, 0)])
def test_w_spread_decides(share, form):
    _, _, part, _, _ = near_the_limit(share)
    assert (pkg.FORM_SINCOS, pkg.FORM_TENSOR_CORE) == (0, 1)
    assert part.plan.info()["device_form"] == form


def still(S, kernel, nt, nch=1):
    """One baseline whose samples all lie at one uv point: one subgrid of nt * nch visibilities."""
    uvw = np.tile([3.0, 5.0, 0.0], (1, nt, 1))
    c = pkg.GriddingConstants(nt * nch, 256, S, kernel, 1024, 1.0 / 4096, 1, 0.0)
    part = pkg.Partitioner.CreatePartition(c, uvw, np.full(nch, 299792458.0))
    assert part.plan.info()["num_subgrids"] == 1 and part.plan.info()["gridded_visibilities"] == nt * nch
    return part.plan


@pytest.mark.parametrize("S,kernel,most_on_sincos", [(16, 4, 375), (24, 8, 107), (32, 8, 53)])
def test_work_per_subgrid_decides(S, kernel, most_on_sincos):
    assert still(S, kernel, most_on_sincos).info()["device_form"] == pkg.FORM_SINCOS
    assert still(S, kernel, most_on_sincos + 1).info()["device_form"] == pkg.FORM_TENSOR_CORE
    assert still(S, kernel, 2, most_on_sincos).info()["device_form"] == pkg.FORM_TENSOR_CORE


def test_sizes_modes_and_the_switch():
    assert still(8, 2, 1000).info()["device_form"] == pkg.FORM_SINCOS
    assert still(48, 8, 1000).info()["device_form"] == pkg.FORM_SINCOS
    plan = still(32, 8, 1000)
    plan.set_fp32_tensor_cores(False)
    assert plan.info()["device_form"] == pkg.FORM_SINCOS
    assert plan.set_mode(pkg.MODE_TC_BF16X3) == pkg.MODE_TC_BF16X3
    assert plan.info()["device_form"] == pkg.FORM_TENSOR_CORE
    plan.set_mode(pkg.MODE_FP32)
    assert plan.info()["device_form"] == pkg.FORM_SINCOS
    plan.set_fp32_tensor_cores(True)
    assert plan.info()["device_form"] == pkg.FORM_TENSOR_CORE


def device_calls(plan, vis, grid, layers_shape):
    import torch

    d_vis, d_grid = torch.from_numpy(vis).cuda(), torch.from_numpy(grid).cuda()
    layers = torch.full(layers_shape, float("nan"), dtype=torch.complex64, device="cuda")
    out = torch.full(vis.shape, float("nan"), dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    plan.grid_w_device(d_vis.data_ptr(), layers.data_ptr())
    plan.degrid_w_device(d_grid.data_ptr(), out.data_ptr())
    plan.synchronize()
    return layers.cpu().numpy(), out.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("share", [0.98, 1.02])
def test_calls_run_the_plans_form(need_gpu, share):
    """The switch changes the degridded bits where the plan runs the tensor cores, and only there; batches too."""
    pytest.importorskip("torch")
    obs, uvw, part, c, d = near_the_limit(share)
    plan, N = part.plan, d["grid_size"]
    tensor = plan.info()["device_form"] == pkg.FORM_TENSOR_CORE
    rng = np.random.default_rng(5)
    grid = (rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))).astype(np.complex64)
    vis = obs.vis.astype(np.complex64)
    shape = (d["wlayer_count"], N, N)
    auto = device_calls(plan, vis, grid, shape)
    plan.set_fp32_tensor_cores(False)
    sincos = device_calls(plan, vis, grid, shape)
    plan.set_fp32_tensor_cores(True)
    again = device_calls(plan, vis, grid, shape)
    assert np.array_equal(auto[1], sincos[1]) == (not tensor)
    assert np.array_equal(auto[1], again[1])
    for a, b in zip(auto, sincos):
        assert rel_l2(a, b) < 1e-5  # both within the FP32 bar of the oracle
