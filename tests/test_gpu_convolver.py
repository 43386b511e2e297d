"""PaddedConvolver over the sizes where its real-to-complex form can go wrong: padded sizes with large
prime factors (transformed at a larger size), odd ones (FFT.Shift keeps the last row and column), images
smaller and larger than the one a correlation was made for, and Fourier kernels that are not Hermitian.

Against the FP64 oracle, whose results are float: 2^-23 of the largest value covers one rounding each.
"""
import numpy as np
import pytest

from conftest import oracle, pkg

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -23


def _close(out, ref):
    assert out.dtype == np.float32 and np.abs(out - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("n,p", [(64, 16), (61, 16), (127, 31), (100, 33), (257, 64), (48, 49), (5, 4), (8, 3)])
def test_correlation(need_gpu, n, p):
    rng = np.random.default_rng(100 * n + p)
    psf = rng.standard_normal((p, p)).astype(np.float32)
    kernel = oracle.padded_fourier_correlation(psf, (n, n))
    conv = pkg.PaddedConvolver.correlation(psf, pkg.Rectangle(0, 0, n, n))
    for m in (n, max(1, n - 3), n + p // 2, n):  # as made for, smaller, the largest that fits, again
        img = rng.standard_normal((m, m)).astype(np.float32)
        _close(conv.Convolve(img), oracle.padded_convolve(kernel, (p, p), img))
    conv.destroy()


@pytest.mark.parametrize("h,ky,kx,n", [(24, 8, 8, 16), (31, 7, 7, 20), (40, 6, 12, 33), (9, 4, 4, 5)])
def test_any_fourier_kernel(need_gpu, h, ky, kx, n):
    rng = np.random.default_rng(h)
    kernel = rng.standard_normal((h, h)) + 1j * rng.standard_normal((h, h))
    img = rng.standard_normal((n, n)).astype(np.float32)
    conv = pkg.PaddedConvolver(kernel, pkg.Rectangle(0, 0, ky, kx))
    _close(conv.Convolve(img), oracle.padded_convolve(kernel, (ky, kx), img))
    conv.destroy()
