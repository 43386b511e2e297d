"""The FP32 mode's device calls on the tensor cores (FP16 operands split hi + lo).

Host-array calls on the same plan run the sincos kernels, so both forms are compared with the FP64
oracle on one plan: the tensor-core form may be no further off than the sincos form.  A tenth of the
sincos form's error is left for the two errors being independent samples, and 1e-7 (about an FP32
unit roundoff of the result and one of the accumulation) for cases where the sincos form's own
error is by chance small.
"""
import numpy as np
import pytest

from conftest import constants, oracle, pkg, rel_l2, workload

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# (S, kernel, channels, times, grid size, degridder / gridder item sizes): one channel, odd grids, items
# that end inside a tile, items split over a subgrid, padded subgrids
SHAPES = [
    (32, 8, 1, 173, 255, None),
    (32, 8, 3, 301, 256, None),
    (32, 8, 16, 131, 512, (320, 384)),
    (24, 8, 5, 301, 257, None),
    (16, 4, 16, 240, 256, (1040, 272)),
]


def _setup(S, kernel, nch, nt, N, chunks):
    obs, cd = workload("small_256", n_ant=9, nt=nt, nch=nch, seed=nch * 100 + nt)
    # the w step a hair above max |w| / layers: with one channel the largest w needs a layer too
    c, cd = constants(cd, grid_size=N, subgrid_size=S, kernel_size=kernel, wstep=cd["wstep"] * (1 + 1e-6))
    part = pkg.Partitioner.CreatePartition(c, obs.uvw, obs.frequencies)
    assert part.plan.info()["mode"] == pkg.MODE_FP32
    if chunks:
        pkg.set_chunking(part.plan, *chunks)
    return obs, c, cd, part, oracle.partition(cd, obs.uvw, obs.frequencies)


def _no_further_off(tc, sincos, ref):
    e_tc, e_sc = rel_l2(tc, ref), rel_l2(sincos, ref)
    print(f"against FP64: tensor cores {e_tc:.2e}, sincos {e_sc:.2e}")
    assert not np.array_equal(tc, sincos.astype(np.complex64))  # two forms ran
    assert e_tc <= 1.1 * e_sc + 1e-7


@pytest.mark.parametrize("S,kernel,nch,nt,N,chunks", SHAPES)
def test_degrid(need_gpu, S, kernel, nch, nt, N, chunks):
    obs, c, cd, part, subs = _setup(S, kernel, nch, nt, N, chunks)
    rng = np.random.default_rng(N)
    model = (rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))).astype(np.complex64)
    d_grid = torch.from_numpy(model).cuda()
    d_out = torch.full(obs.vis.shape, float("nan"), dtype=torch.complex64, device="cuda")
    part.plan.degrid_w_device(d_grid.data_ptr(), d_out.data_ptr())
    part.plan.synchronize()
    host = pkg.IDG.DeGridW(c, part, model.astype(np.complex128), obs.uvw, obs.frequencies)
    ref, _ = oracle.idg_degrid(cd, subs, model.astype(np.complex128), obs.uvw, obs.frequencies, wstack=True)
    _no_further_off(d_out.cpu().numpy(), host, ref)


@pytest.mark.parametrize("S,kernel,nch,nt,N,chunks", SHAPES)
def test_grid(need_gpu, S, kernel, nch, nt, N, chunks):
    obs, c, cd, part, subs = _setup(S, kernel, nch, nt, N, chunks)
    vis = obs.vis.astype(np.complex64)
    d_vis = torch.from_numpy(vis).cuda()
    d_layers = torch.full((cd["wlayer_count"], N, N), float("nan"), dtype=torch.complex64, device="cuda")
    part.plan.grid_w_device(d_vis.data_ptr(), d_layers.data_ptr())
    part.plan.synchronize()
    host = pkg.IDG.GridW(c, part, vis.astype(np.complex128), obs.uvw, obs.frequencies)
    ref = oracle.idg_grid_w(cd, subs, vis.astype(np.complex128), obs.uvw, obs.frequencies)
    _no_further_off(d_layers.cpu().numpy(), host, ref)
