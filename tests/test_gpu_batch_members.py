"""A batch keeps the form its plans had when it was made, whatever is done to a plan afterwards."""
import numpy as np
import pytest

from conftest import constants, pkg, rel_l2, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _problems(mode, sizes):
    out = []
    for i, (S, kernel, N) in enumerate(sizes):
        obs, cd = synth.build(synth.scaled_workload("small_256", n_ant=6 + i, nt=160 + 40 * i, nch=4 + 2 * i, seed=31 + i))
        c, cd = constants(cd, grid_size=N, subgrid_size=S, kernel_size=kernel)
        part = pkg.Partitioner.CreatePartition(c, obs.uvw, obs.frequencies)
        assert part.plan.set_mode(mode) == mode
        g = torch.Generator(device="cuda").manual_seed(i)
        out.append((part, c, obs, dict(
            vis=torch.from_numpy(obs.vis.astype(np.complex64)).cuda(),
            layers=torch.empty((cd["wlayer_count"], N, N), dtype=torch.complex64, device="cuda"),
            grid=torch.randn((N, N), dtype=torch.complex64, device="cuda", generator=g),
            out=torch.empty(obs.vis.shape, dtype=torch.complex64, device="cuda"))))
    torch.cuda.synchronize()
    return out


def _batch(probs):
    ptr = lambda k: [b[k].data_ptr() for _, _, _, b in probs]  # noqa: E731
    return pkg.Batch([p.plan for p, _, _, _ in probs], ptr("vis"), ptr("layers"), ptr("grid"), ptr("out"))


def _run(batch, probs):
    for _, _, _, b in probs:
        b["layers"].fill_(float("nan"))
        b["out"].fill_(float("nan"))
    torch.cuda.synchronize()
    batch.run()
    batch.synchronize()
    return [(b["layers"].cpu().numpy(), b["out"].cpu().numpy()) for _, _, _, b in probs]


def _same(got, ref):
    for (layers, vis), (rl, rv) in zip(got, ref):
        # the adder's FP32 atomics add in any order: a few units of 6e-8
        assert rel_l2(layers, rl) < 1e-6
        assert rel_l2(vis, rv) < 1e-6


# S = 8 keeps the sincos kernels in the FP32 mode, so the change of mode changes the first plan's form: it is
# alone in its group, or shares it with a plan that stays as it is.
@pytest.mark.parametrize("mode,other", [(pkg.MODE_FP32, pkg.MODE_TC_BF16X3), (pkg.MODE_TC_BF16X3, pkg.MODE_FP32)],
                         ids=["fp32", "bf16x3"])
@pytest.mark.parametrize("sizes", [[(8, 2, 256), (32, 8, 256)], [(8, 2, 256), (8, 2, 300), (16, 4, 256)]],
                         ids=["two_sizes", "shared_size"])
def test_member_changes_mode_then_schedule(need_gpu, mode, other, sizes):
    probs = _problems(mode, sizes)
    batch = _batch(probs)
    ref = _run(batch, probs)
    assert probs[0][0].plan.set_mode(other) == other
    batch.set_schedule(pkg.Batch.SMALL_FIRST)
    _same(_run(batch, probs), ref)
    batch.capture_graph()
    _same(_run(batch, probs), ref)
    batch.destroy()


def test_member_needs_more_partial_subgrids_of_its_own(need_gpu):
    """The plan's own calls with smaller work items, in another mode and in the batch's, between runs and replays
    of the batch: they need more partial subgrids than the batch does, in memory that the batch does not use."""
    probs = _problems(pkg.MODE_TC_BF16X3, [(32, 8, 256), (16, 4, 300)])
    batch = _batch(probs)
    batch.capture_graph()
    ref = _run(batch, probs)
    for part, c, obs, b in probs:
        plan = part.plan
        slots = plan.info()["work_items"]
        pkg.set_chunking(plan, 64, 64)
        assert plan.info()["work_items"] > 4 * slots
        lay, vis = torch.empty_like(b["layers"]), torch.empty_like(b["out"])
        plan.grid_w_device(b["vis"].data_ptr(), lay.data_ptr())
        plan.degrid_w_device(b["grid"].data_ptr(), vis.data_ptr())
        plan.synchronize()
        assert plan.set_mode(pkg.MODE_FP32) == pkg.MODE_FP32
        pkg.IDG.GridW(c, part, obs.vis, obs.uvw, obs.frequencies)
        # what the plans gave back is used by others, as a program's next allocation would
        junk = [torch.full((1 << 20,), float("nan"), device="cuda") for _ in range(32)]
    _same(_run(batch, probs), ref)
    batch.set_schedule(pkg.Batch.SMALL_FIRST)
    _same(_run(batch, probs), ref)
    del junk
    batch.destroy()
