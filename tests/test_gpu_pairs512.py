"""The 512-point kernels on pairs (pairs512.cuh): the fused z pass against a real filter's half
spectrum, a complex filter and a given spectrum, and the real filter's x pass.

One convolution of two signals against FP64 by all three routes; the signals differ in
scale, the filter is neither symmetric nor smooth. Tolerance: the reference's criterion, a
relative L2 error of 1e-6 (the FP32 passes are at 3-4e-7).
"""
import numpy as np
import pytest

from oracle import conv3d, rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
N, HERM = 512, 7


def test_routes(gpu):
    rng = np.random.default_rng(512)
    sig = rng.standard_normal((2, N, N, N, 2), dtype=np.float32).view(np.complex64)[..., 0]
    sig[1] *= 100
    filt = rng.standard_normal((N, N, N), dtype=np.float32)
    s, f = torch.from_numpy(sig).cuda(), torch.from_numpy(filt).cuda()
    spec = torch.empty((N, N, N), dtype=torch.complex64, device="cuda")
    gpu.filter_spectrum_device(N, f.to(torch.complex64), spec, 1)
    ref = [conv3d(sig[i:i + 1], filt.astype(np.complex64), "fp64", engine="pocketfft")[0] for i in (1,)][0]
    keep = gpu.plan_variant(N, HERM)
    gpu.device_status()
    outs = []
    for herm, filter_, flags in ((1, f, gpu.FILTER_REAL), (0, f.to(torch.complex64), 0), (0, spec, gpu.FILTER_IS_SPECTRUM)):
        gpu.plan_variant(N, HERM, herm)
        o = torch.empty_like(s)
        gpu.conv3d_device(N, s, filter_, o, 2, flags)
        torch.cuda.synchronize()
        assert rel_l2(ref, o[1].cpu().numpy()) < 1e-6, flags
        outs.append(o[0])
    gpu.plan_variant(N, HERM, keep)
    assert gpu.device_status() == 0
    # the first signal, to twice the tolerance of each against the others
    for o in outs[1:]:
        assert float(torch.linalg.vector_norm(o - outs[0]) / torch.linalg.vector_norm(outs[0])) < 2e-6


@pytest.mark.parametrize("shift", [(0, 0, 0), (3, 511, 257), (256, 256, 256), (1, 8, 504)])
def test_impulse_reproduces_filter(gpu, shift):
    """Rows y and -y, columns x and -x, the self-mirrored ones: all land where they belong."""
    keep = gpu.plan_variant(N, HERM)
    gpu.plan_variant(N, HERM, 1)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(sum(shift))
    f = torch.randn((N, N, N), generator=gen, device="cuda")
    s = torch.zeros((1, N, N, N), dtype=torch.complex64, device="cuda")
    s[0][shift] = 1.0
    gpu.conv3d_device(N, s, f, s, 1, gpu.FILTER_REAL | gpu.NORMALIZE)
    torch.cuda.synchronize()
    gpu.plan_variant(N, HERM, keep)
    want = torch.roll(f, shift, (0, 1, 2))
    assert float(torch.linalg.vector_norm(s[0] - want) / torch.linalg.vector_norm(want)) < 1e-6
