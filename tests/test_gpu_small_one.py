"""One cube of N = 32 or 64 in one cooperative launch (k_tp_one, twopass.cuh): complex and real
filters, 8-byte aligned operands, in place, the filter in the output's memory, and a call
captured into a graph, all against the oracle. Tolerance: 120 dB against FP32 and a relative
L2 error of 1e-6 against FP64 (the FP32 passes are at 3e-7)."""
import numpy as np
import pytest

from oracle import conv3d, rel_l2, snr_db

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _c64(rng, shape):
    a = np.empty(shape, np.complex64)
    a.real = rng.uniform(-1, 1, shape)
    a.imag = rng.uniform(-1, 1, shape)
    return a


@pytest.mark.parametrize("n", [32, 64])
@pytest.mark.parametrize("how", ["apart", "unaligned", "in_place", "filter_in_out", "real", "captured"])
def test_one_cube(gpu, n, how):
    rng = np.random.default_rng(n)
    sig, filt = _c64(rng, (n, n, n)), _c64(rng, (n, n, n))
    if how == "real":
        filt.imag = 0
    off = 1 if how == "unaligned" else 0

    def dev(a):
        t = torch.empty(a.size + off, dtype=torch.complex64, device="cuda")[off:]
        return t.copy_(torch.from_numpy(a).flatten())

    s, f = dev(sig), dev(filt)
    o = s if how == "in_place" else (f if how == "filter_in_out" else dev(np.zeros_like(sig)))
    gpu.device_status()
    if how == "real":
        gpu.conv3d_device(n, s, torch.from_numpy(filt.real.copy()).cuda(), o, 1, gpu.NORMALIZE | gpu.FILTER_REAL)
    elif how == "captured":
        gpu.conv3d_device(n, s, f, o, 1, gpu.NORMALIZE)
        torch.cuda.synchronize()
        o.zero_()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            gpu.conv3d_device(n, s, f, o, 1, gpu.NORMALIZE, torch.cuda.current_stream())
        for k in (3, 2, 1):  # replays on changed data
            s.copy_(torch.from_numpy(k * sig).flatten())
            g.replay()
    else:
        gpu.conv3d_device(n, s, f, o, 1, gpu.NORMALIZE)
    torch.cuda.synchronize()
    assert gpu.device_status() == 0
    out = o.cpu().numpy().reshape(n, n, n)
    assert snr_db(conv3d(sig, filt, "fp32", normalize=True, engine="pocketfft"), out) > 120.0
    assert rel_l2(conv3d(sig, filt, "fp64", normalize=True, engine="pocketfft"), out) < 1e-6
