"""Device calls captured into a CUDA graph keep their buffers when the plan's other calls run between replays."""
import numpy as np
import pytest

from conftest import constants, pkg, rel_l2, workload

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MODES = [pytest.param(pkg.MODE_FP32, id="fp32"), pytest.param(pkg.MODE_TC_BF16X3, id="bf16x3")]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("N", [256, 500])
def test_replay_after_host_calls(need_gpu, mode, N):
    obs, cd = workload("small_256", n_ant=9, nt=300, nch=8)
    c, cd = constants(cd, grid_size=N)
    part = pkg.Partitioner.CreatePartition(c, obs.uvw, obs.frequencies)
    plan = part.plan
    assert plan.set_mode(mode) == mode
    stream = torch.cuda.Stream()
    plan.set_stream(stream.cuda_stream)
    vis = torch.from_numpy(obs.vis.astype(np.complex64)).cuda()
    model = np.random.default_rng(N).standard_normal((N, N)) + 0j
    grid = torch.from_numpy(model.astype(np.complex64)).cuda()
    layers = torch.empty((cd["wlayer_count"], N, N), dtype=torch.complex64, device="cuda")
    image = torch.empty((N, N), device="cuda")
    out = torch.empty_like(vis)
    torch.cuda.synchronize()

    def calls():
        plan.grid_w_device(vis.data_ptr(), layers.data_ptr())
        plan.wstack_image_device(layers.data_ptr(), image.data_ptr())
        plan.degrid_w_device(grid.data_ptr(), out.data_ptr())

    calls()
    plan.synchronize()
    ref = [t.cpu().numpy() for t in (layers, image, out)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        calls()
    for t in (layers, image, out):
        t.fill_(float("nan"))
    # every other call that uses the plan's buffers, then allocations that take up what they gave back
    pkg.IDG.GridW(c, part, obs.vis, obs.uvw, obs.frequencies)
    pkg.IDG.DeGridW(c, part, model.copy(), obs.uvw, obs.frequencies)
    plan.set_host_access(False)
    pkg.IDG.GridW(c, part, obs.vis, obs.uvw, obs.frequencies)
    pkg.IDG.DeGridW(c, part, model.copy(), obs.uvw, obs.frequencies)
    junk = [torch.full((1 << 20,), float("nan"), device="cuda") for _ in range(32)]
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        graph.replay()
    torch.cuda.synchronize()
    plan.synchronize()
    for t, r in zip((layers, image, out), ref):
        # the adder's FP32 atomics add in any order
        assert rel_l2(t.cpu().numpy(), r) < 1e-6
    del junk


@pytest.mark.parametrize("chunks", [None, (512, 1024)], ids=["default", "set"])
def test_replay_after_a_change_of_mode_and_back(need_gpu, chunks):
    """The modes cut a small observation into different work items; a graph captured from one mode's calls finds
    its own again once the plan is back in that mode."""
    obs, cd = workload("small_256", n_ant=9, nt=300, nch=8)
    c, cd = constants(cd)
    N = cd["grid_size"]
    part = pkg.Partitioner.CreatePartition(c, obs.uvw, obs.frequencies)
    plan = part.plan
    if chunks:
        pkg.set_chunking(plan, *chunks)
    stream = torch.cuda.Stream()
    plan.set_stream(stream.cuda_stream)
    vis = torch.from_numpy(obs.vis.astype(np.complex64)).cuda()
    grid = torch.randn((N, N), dtype=torch.complex64, device="cuda")
    layers = torch.empty((cd["wlayer_count"], N, N), dtype=torch.complex64, device="cuda")
    out = torch.empty_like(vis)
    torch.cuda.synchronize()

    def calls(mode):
        assert plan.set_mode(mode) == mode
        plan.grid_w_device(vis.data_ptr(), layers.data_ptr())
        plan.degrid_w_device(grid.data_ptr(), out.data_ptr())
        plan.synchronize()

    modes = (pkg.MODE_FP32, pkg.MODE_TC_BF16X3)
    for mode in modes:  # every buffer at its largest
        calls(mode)
    for mode in modes:
        other = modes[1 - modes.index(mode)]
        calls(mode)
        ref = [t.cpu().numpy() for t in (layers, out)]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            plan.grid_w_device(vis.data_ptr(), layers.data_ptr())
            plan.degrid_w_device(grid.data_ptr(), out.data_ptr())
        calls(other)
        junk = [torch.full((1 << 18,), float("nan"), device="cuda") for _ in range(32)]
        calls(mode)
        layers.fill_(float("nan"))
        out.fill_(float("nan"))
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            graph.replay()
        torch.cuda.synchronize()
        plan.synchronize()
        for t, r in zip((layers, out), ref):
            assert rel_l2(t.cpu().numpy(), r) < 1e-6
        del junk
