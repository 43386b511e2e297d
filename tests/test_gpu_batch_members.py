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
