"""What a change of mode costs the next call: nothing that the mode does not change.

The launches of a call are counted in a stream capture (the driver API, by ctypes).
"""
import ctypes

import numpy as np
import pytest

from conftest import constants, oracle, pkg, rel_l2, workload

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _launches(stream, call):
    cu = ctypes.CDLL("libcuda.so.1")
    s, graph, n = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p(), ctypes.c_size_t()
    assert cu.cuStreamBeginCapture_v2(s, 1) == 0  # this thread's calls
    try:
        call()
    finally:
        rc = cu.cuStreamEndCapture(s, ctypes.byref(graph))
    assert rc == 0
    assert cu.cuGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    assert cu.cuGraphDestroy(graph) == 0
    return n.value


def test_coefficients_survive_a_change_of_mode(need_gpu):
    obs, cd = workload("small_256", n_ant=8, nt=200, nch=8)
    c, cd = constants(cd)
    N = cd["grid_size"]
    part = pkg.Partitioner.CreatePartition(c, obs.uvw, obs.frequencies)
    plan = part.plan
    stream = torch.cuda.Stream()
    plan.set_stream(stream.cuda_stream)
    rng = np.random.default_rng(4)
    model = (rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))).astype(np.complex64)
    grid = torch.from_numpy(model).cuda()
    out = torch.empty(obs.vis.shape, dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    subs = oracle.partition(cd, obs.uvw, obs.frequencies)
    ref, _ = oracle.idg_degrid(cd, subs, model.astype(np.complex128), obs.uvw, obs.frequencies, wstack=True)

    def call():
        plan.degrid_w_device(grid.data_ptr(), out.data_ptr())

    for mode in (pkg.MODE_TC_BF16X3, pkg.MODE_TC_FP16X3):
        plan.set_mode(mode)
        call()
        plan.synchronize()
    usual = _launches(stream, call)
    assert usual >= 2  # splitter and degridder
    for mode in (pkg.MODE_TC_BF16X3, pkg.MODE_TC_FP16X3):
        plan.set_mode(mode)
        assert _launches(stream, call) == usual
    # through the FP32 mode, whose coefficients are not checked, and a host call with another uvw
    other = obs.uvw * np.array([1.0, 1.0, 0.5])
    for mode, bound in ((pkg.MODE_FP32, 1e-5), (pkg.MODE_TC_BF16X3, 1e-4), (pkg.MODE_FP32, 1e-5),
                        (pkg.MODE_TC_FP16X3, 1e-4)):
        assert plan.set_mode(mode) == mode
        call()
        plan.synchronize()
        assert rel_l2(out.cpu().numpy(), ref) < bound
        pkg.IDG.DeGridW(c, part, model.astype(np.complex128), other, obs.frequencies)
