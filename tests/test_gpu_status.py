"""Who reports a tripped check: the call that tripped it, or the synchronisation after it, once.

The checks are made to trip by the bounded waits' fault injection (p9idg_debug_tc_wait): a 1 ms limit and a
loader that never delivers input stage 1 of its work items.
"""
import numpy as np
import pytest

from conftest import constants, oracle, pkg, rel_l2, workload

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
CHECK_FAILED = 9


class _Injected:
    def __enter__(self):
        assert pkg._native.lib().p9idg_debug_tc_wait(1_000_000, 1) == 0

    def __exit__(self, *a):
        assert pkg._native.lib().p9idg_debug_tc_wait(0, -1) == 0


def _problem(seed=0):
    obs, cd = workload("small_256", n_ant=8, nt=300, nch=8)
    c, cd = constants(cd)
    part = pkg.Partitioner.CreatePartition(c, obs.uvw, obs.frequencies)
    assert part.plan.set_mode(pkg.MODE_TC_BF16X3) == pkg.MODE_TC_BF16X3
    N = cd["grid_size"]
    vis = torch.from_numpy(obs.vis.astype(np.complex64)).cuda()
    layers = torch.empty((cd["wlayer_count"], N, N), dtype=torch.complex64, device="cuda")
    grid = torch.randn((N, N), dtype=torch.complex64, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
    torch.cuda.synchronize()
    return obs, c, cd, part, dict(vis=vis, layers=layers, grid=grid, out=torch.empty_like(vis))


def _fails(call):
    with pytest.raises(pkg.P9IDGError) as e:
        call()
    assert e.value.code == CHECK_FAILED
    return str(e.value)


def _flags(obs):
    return np.zeros(obs.vis.shape, np.uint8)


def test_device_call_then_host_call_then_synchronize(need_gpu):
    obs, c, cd, part, b = _problem()
    plan = part.plan
    subs = oracle.partition(cd, obs.uvw, obs.frequencies)
    ref = oracle.idg_grid_w(cd, subs, obs.vis, obs.uvw, obs.frequencies)
    for uvw in (obs.uvw, None):
        with _Injected():
            plan.grid_w_device(b["vis"].data_ptr(), b["layers"].data_ptr())
        # the host calls between report their own checks only, whichever uvw they pass ...
        assert rel_l2(pkg.IDG.GridW(c, part, obs.vis, uvw, obs.frequencies), ref) < 1e-4
        pkg.IDG.GridPSF(c, part, uvw, _flags(obs), obs.frequencies)
        # ... and the device call's is still there, to be reported once
        _fails(plan.synchronize)
        plan.synchronize()


def test_host_call_reports_its_own(need_gpu):
    obs, c, cd, part, b = _problem()
    with _Injected():
        _fails(lambda: pkg.IDG.GridW(c, part, obs.vis, obs.uvw, obs.frequencies))
    part.plan.synchronize()
    part.plan.grid_w_device(b["vis"].data_ptr(), b["layers"].data_ptr())
    part.plan.synchronize()


def test_batch_reports_every_problem_once(need_gpu):
    probs = [_problem(i) for i in range(3)]
    ptr = lambda k: [p[4][k].data_ptr() for p in probs]  # noqa: E731
    plans = [p[3].plan for p in probs]
    with _Injected():  # a batch keeps the injection it was made with
        batch = pkg.Batch(plans, ptr("vis"), ptr("layers"), ptr("grid"), ptr("out"))
    batch.run()
    assert "problem 0" in _fails(batch.synchronize)
    batch.synchronize()
    for p in plans:  # nothing of the batch is left for the plans' own reports
        p.synchronize()
    # and a plan's own failure is reported by the plan
    with _Injected():
        plans[1].grid_w_device(probs[1][4]["vis"].data_ptr(), probs[1][4]["layers"].data_ptr())
    batch.synchronize()
    plans[0].synchronize()
    _fails(plans[1].synchronize)
    batch.destroy()


def test_refused_uvw_is_refused_again(need_gpu):
    """A uvw beyond the tensor-core form's w bound is refused however often it is passed."""
    from test_tc_w_term import wide_field

    obs, uvw, c, d = wide_field(0.5 * pkg.TC_MAX_W_TERM)
    part = pkg.Partitioner.CreatePartition(c, uvw, obs.frequencies)
    assert part.plan.set_mode(pkg.MODE_TC_BF16X3) == pkg.MODE_TC_BF16X3
    big = uvw.copy()
    big[..., 2] *= 3.0
    pkg.IDG.GridW(c, part, obs.vis, uvw, obs.frequencies)
    for _ in range(3):
        with pytest.raises(pkg.P9IDGError) as e:
            pkg.IDG.GridW(c, part, obs.vis, big, obs.frequencies)
        assert e.value.code == 8
    pkg.IDG.GridW(c, part, obs.vis, uvw, obs.frequencies)
