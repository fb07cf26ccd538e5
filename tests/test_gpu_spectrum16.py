"""Forward transforms of 16^3 cubes in one launch (k_spectrum16, cube16.cu): odd and even counts,
8-byte aligned, in place. Tolerance: a relative L2 error of 1e-6 against FP64, the bound of
the other FP32 transforms (2-3e-7 measured)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("count", [1, 2, 5, 301])
@pytest.mark.parametrize("how", ["apart", "unaligned", "in_place"])
def test_spectra(gpu, count, how):
    rng = np.random.default_rng(count)
    a = (rng.standard_normal((count, 16, 16, 16)) + 1j * rng.standard_normal((count, 16, 16, 16))).astype(np.complex64)
    off = 1 if how == "unaligned" else 0
    x = torch.zeros(a.size + 8, dtype=torch.complex64, device="cuda")
    x[off:off + a.size] = torch.from_numpy(a).flatten().cuda()
    y = x if how == "in_place" else torch.zeros_like(x)
    l0 = gpu.launch_count()
    gpu.filter_spectrum_device(16, x[off:], y[off:], count)
    torch.cuda.synchronize()
    assert gpu.launch_count() - l0 == 1
    got = y[off:off + a.size].cpu().numpy().reshape(a.shape)
    want = np.fft.fftn(a.astype(np.complex128), axes=(1, 2, 3))
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < 1e-6
    assert not y[off + a.size:].abs().any()
