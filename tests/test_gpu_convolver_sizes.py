"""A correlation that has met an image larger than it was made for goes on serving the others as before."""
import time

import numpy as np
import pytest

from conftest import oracle, pkg

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TOL = 2.0 ** -23  # float results of FP64 transforms
OOM = 5


def _arm(after):
    assert pkg._native.lib().p9idg_debug_fail_device_allocations(after) == 0


@pytest.mark.parametrize("failing", [0, 1, 2, 3])
def test_no_memory_for_the_larger_size(need_gpu, failing):
    """Each allocation of the padded size's transforms fails in turn: the call reports it, and both sizes work
    afterwards."""
    n, p = 127, 31
    rng = np.random.default_rng(failing)
    psf = rng.standard_normal((p, p)).astype(np.float32)
    kernel = oracle.padded_fourier_correlation(psf, (n, n))
    conv = pkg.PaddedConvolver.correlation(psf, pkg.Rectangle(0, 0, n, n))
    img = {m: torch.from_numpy(rng.standard_normal((m, m)).astype(np.float32)).cuda() for m in (n, n + p // 2)}
    out = {m: torch.empty_like(img[m]) for m in img}
    ref = {m: oracle.padded_convolve(kernel, (p, p), img[m].cpu().numpy()) for m in img}
    torch.cuda.synchronize()

    def check(m):
        out[m].fill_(float("nan"))
        torch.cuda.synchronize()
        conv.convolve_device(img[m].data_ptr(), m, out[m].data_ptr())
        torch.cuda.synchronize()
        assert np.abs(out[m].cpu().numpy() - ref[m]).max() <= TOL * np.abs(ref[m]).max()

    check(n)
    _arm(failing)
    try:
        with pytest.raises(pkg.P9IDGError) as e:
            conv.convolve_device(img[n + p // 2].data_ptr(), n + p // 2, out[n + p // 2].data_ptr())
        assert e.value.code == OOM
    finally:
        _arm(-1)
    for m in (n, n + p // 2, n, n + p // 2):
        check(m)
    conv.destroy()


def test_the_made_size_stays_fast(need_gpu):
    """1279 + 128 = 1407 = 3 * 7 * 67: the padded size's transforms take several times the next even 7-smooth one's."""
    n, p = 1279, 128
    psf = np.random.default_rng(1).standard_normal((p, p)).astype(np.float32)
    conv = pkg.PaddedConvolver.correlation(psf, pkg.Rectangle(0, 0, n, n))
    big = torch.randn((n + p // 2, n + p // 2), device="cuda")
    img, out = big[:n, :n].contiguous(), torch.empty_like(big)

    def seconds(a, m):
        best = 1e9
        for _ in range(8):
            torch.cuda.synchronize()
            t = time.perf_counter()
            for _ in range(4):
                conv.convolve_device(a.data_ptr(), m, out.data_ptr())
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        return best

    before = seconds(img, n)
    large = seconds(big, n + p // 2)
    after = seconds(img, n)
    print(f"made for {before * 250:.3f} ms, larger {large * 250:.3f} ms, made for again {after * 250:.3f} ms")
    assert large > 1.5 * before  # else this size shows nothing
    assert after < 1.2 * before
    conv.destroy()
