"""The FP32 mode's tensor-core form is no further from FP64 than the sincos kernels, on skies of all kinds.

Both forms run as device calls of one plan.  Degridding has no atomics, and its error is an average over tens
of thousands of visibilities (a spread below 1 %).  A gridded layer's error moves by some 20 % from run to run, as
the adder's FP32 atomics meet in another order in the few brightest pixels: the mean of four runs of each form is
taken, which leaves 10 % each and 1.15 for their ratio.
"""
import numpy as np
import pytest

from conftest import oracle, pkg, rel_l2
from test_fp32_form import device_calls, near_the_limit

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _sky(name, vis):
    rng = np.random.default_rng(11)
    if name == "noise":
        return rng.standard_normal(vis.shape) + 1j * rng.standard_normal(vis.shape)
    if name == "sparse":  # one visibility in 64, so that a tensor-core sum holds one of them
        return vis * (rng.random(vis.shape) < 1 / 64)
    if name == "outliers":
        return np.where(rng.random(vis.shape) < 1 / 500, 1e4, 1.0) * vis
    return vis if name == "sources" else np.ones(vis.shape)


@pytest.mark.parametrize("share", [0.25, 0.98])
@pytest.mark.parametrize("sky", ["sources", "noise", "sparse", "outliers", "ones"])
def test_no_further_off_than_sincos(need_gpu, sky, share):
    obs, uvw, part, c, d = near_the_limit(share)
    plan, N = part.plan, d["grid_size"]
    assert plan.info()["device_form"] == pkg.FORM_TENSOR_CORE
    vis = _sky(sky, obs.vis).astype(np.complex64)
    rng = np.random.default_rng(7)
    grid = (np.ones((N, N)) if sky == "ones" else rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N)))
    grid = grid.astype(np.complex64)
    subs = oracle.partition(d, uvw, obs.frequencies)
    layers = oracle.idg_grid_w(d, subs, vis.astype(np.complex128), uvw, obs.frequencies)
    model, _ = oracle.idg_degrid(d, subs, grid.astype(np.complex128), uvw, obs.frequencies, wstack=True)
    err = {}
    for on in (True, False):
        plan.set_fp32_tensor_cores(on)
        runs = [device_calls(plan, vis, grid, layers.shape) for _ in range(4)]
        err[on] = (np.mean([rel_l2(g, layers) for g, _ in runs]), rel_l2(runs[0][1], model))
    print(f"{sky}: tensor cores {err[True]}, sincos {err[False]}")
    assert err[True][0] <= 1.15 * err[False][0]
    assert err[True][1] <= 1.01 * err[False][1]
