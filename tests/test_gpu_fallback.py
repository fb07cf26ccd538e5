"""Which passes run the calls that the two-pass transform does not take (plan kind 4, variant 3):
separate passes up to five cubes of 128^3, the staged pass beyond and at 256^3. Told apart by
the passes that are timed; the results against numpy's FFT at 64 bits (1e-6, the criterion of the
FP32 passes)."""
import numpy as np
import pytest

from oracle import rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,b,staged", [(128, 1, False), (128, 5, False), (128, 6, True), (128, 9, True), (256, 1, True),
                                        (64, 3, False)])
def test_spectra(gpu, n, b, staged):
    keep = gpu.plan_variant(n, 4)
    gpu.plan_variant(n, 4, 3)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n + b)
    f = torch.view_as_complex(torch.randn((b, n, n, n, 2), generator=gen, device="cuda"))
    spec = torch.empty_like(f)
    try:
        gpu.filter_spectrum_device(n, f, spec, b)  # allocations
        gpu.pass_timing_start()
        gpu.filter_spectrum_device(n, f, spec, b)
        torch.cuda.synchronize()
        passes = gpu.pass_timing_read()
        gpu.pass_timing_stop()
        assert set(passes) == ({"xy-fwd", "z-fwd"} if staged else {"x-fwd", "y-fwd", "z-fwd"})
        for i in {0, b - 1}:
            assert rel_l2(np.fft.fftn(f[i].cpu().numpy().astype(np.complex128)), spec[i].cpu().numpy()) < 1e-6
    finally:
        gpu.plan_variant(n, 4, keep)


@pytest.mark.parametrize("n,b,tiles", [(32, 1, True), (32, 47, True), (32, 48, False), (32, 299, False), (32, 300, True),
                                       (64, 8, True), (64, 9, False), (64, 31, False), (64, 32, True)])
def test_signals_against_a_spectrum(gpu, n, b, tiles):
    """Tiles (reordering, forward, middle, inverse) or separate passes (x, y, z, y, x)."""
    keep = gpu.plan_variant(n, 4)
    gpu.plan_variant(n, 4, 3)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n + b)
    s = torch.view_as_complex(torch.randn((b, n, n, n, 2), generator=gen, device="cuda"))
    spec = torch.view_as_complex(torch.randn((n, n, n, 2), generator=gen, device="cuda"))
    o = torch.empty_like(s)
    try:
        gpu.conv3d_device(n, s, spec, o, b, gpu.FILTER_IS_SPECTRUM)  # allocations
        before = gpu.launch_count()
        gpu.conv3d_device(n, s, spec, o, b, gpu.FILTER_IS_SPECTRUM | gpu.NORMALIZE)
        assert gpu.launch_count() - before == (4 if tiles else 5)
        torch.cuda.synchronize()
        f = spec.cpu().numpy().astype(np.complex128)
        for i in {0, b - 1}:
            ref = np.fft.ifftn(np.fft.fftn(s[i].cpu().numpy().astype(np.complex128)) * f)
            assert rel_l2(ref, o[i].cpu().numpy()) < 1e-6
        assert gpu.device_status() == 0
    finally:
        gpu.plan_variant(n, 4, keep)
