"""The w layers' image (FFT.WStackIFFTFloat and its device form) by a complex-to-real transform: even and
odd grids, shifted and not, one layer and several, outputs at addresses the transform cannot write.

Against numpy in FP64.  The transform's single-precision rounding grows with its log2(n^2) passes and the
layers' sum adds one rounding per layer: each at most 2^-24 of the values' norm.
"""
import numpy as np
import pytest

from conftest import oracle, pkg, rel_l2, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SIZES = [(32, 1), (33, 2), (63, 3), (64, 8), (130, 5), (257, 1)]


def _bound(n, w):
    return (2 * np.log2(n) + w + 1) * 2.0 ** -24


def _layers(n, w):
    rng = np.random.default_rng(1000 * n + w)
    return (rng.standard_normal((w, n, n)) + 1j * rng.standard_normal((w, n, n))).astype(np.complex64)


def _reference(layers, vis_count):
    n = layers.shape[-1]
    return np.fft.ifft2(layers.astype(np.complex128).sum(0)).real * (n * n / vis_count)


@pytest.mark.parametrize("n,w", SIZES)
def test_device(need_gpu, n, w):
    layers = _layers(n, w)
    c = pkg.GriddingConstants(777, n, 8, 2, 16, synth.cell_rad(1.5), w, 0.0)
    plan = pkg.Partitioner.CreatePartition(c, np.zeros((1, 1, 3)), np.array([1.2e9])).plan
    d = torch.from_numpy(layers).cuda()
    ref = _reference(layers, 777)
    for shift in (False, True):
        for at in (0, 1):  # elements past an aligned address
            out = torch.full((n * n + 1,), float("nan"), device="cuda")
            torch.cuda.synchronize()
            plan.wstack_image_device(d.data_ptr(), out[at:].data_ptr(), shift)
            plan.synchronize()
            got = out[at:at + n * n].cpu().numpy().reshape(n, n)
            want = oracle.shift(ref.copy()) if shift else ref
            assert rel_l2(got, want) < _bound(n, w)
            assert np.isnan(out.cpu().numpy()).sum() == 1  # the image and nothing else was written
    assert torch.equal(d.cpu(), torch.from_numpy(layers))


@pytest.mark.parametrize("n,w", SIZES)
def test_host(need_gpu, n, w):
    layers = _layers(n, w).astype(np.complex128)
    assert rel_l2(pkg.FFT.WStackIFFTFloat(layers, 777), _reference(layers, 777)) < _bound(n, w)
