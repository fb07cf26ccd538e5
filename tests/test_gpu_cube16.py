"""16^3 convolutions in one launch, one CTA per cube (cube16.cu): every filter kind, batches
from one cube to more than one wave of CTAs, in place, filters in the outputs' memory, the
uneven graph's table mode. Tolerance: the reference's 120 dB criterion and 1e-6 relative L2
against FP64."""
import numpy as np
import pytest

from oracle import conv3d, rel_l2, snr_db

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
N = 16


def _c64(rng, shape):
    a = np.empty(shape, np.complex64)
    a.real = rng.uniform(-1, 1, shape)
    a.imag = rng.uniform(-1, 1, shape)
    return a


def _check(sig, f, out, normalize):
    for i in {0, len(sig) // 2, len(sig) - 1}:
        fi = f[i] if f.ndim == 4 else f
        assert snr_db(conv3d(sig[i:i + 1], fi, "fp32", normalize=normalize)[0], out[i]) > 120.0
        assert rel_l2(conv3d(sig[i:i + 1], fi, "fp64", normalize=normalize)[0], out[i]) < 1e-6


@pytest.mark.parametrize("filt", ["shared", "pairs", "real", "real_pairs", "spectrum", "spectrum_pairs"])
@pytest.mark.parametrize("b", [1, 5, 400])
def test_filter_kinds(gpu, b, filt):
    rng = np.random.default_rng(b)
    sig = _c64(rng, (b, N, N, N))
    f = _c64(rng, (b, N, N, N) if filt.endswith("pairs") else (N, N, N))
    flags = gpu.NORMALIZE | (gpu.FILTER_PER_SIGNAL if filt.endswith("pairs") else 0)
    if filt.startswith("real"):
        f, flags = f.real.copy(), flags | gpu.FILTER_REAL
    s, d = torch.from_numpy(sig).cuda(), torch.from_numpy(f).cuda()
    if filt.startswith("spectrum"):
        spec = torch.empty_like(d)
        gpu.filter_spectrum_device(N, d, spec, b if filt.endswith("pairs") else 1)
        d, flags = spec, flags | gpu.FILTER_IS_SPECTRUM
    o = torch.empty_like(s)
    l0 = gpu.launch_count()
    gpu.conv3d_device(N, s, d, o, b, flags)
    assert gpu.launch_count() - l0 == 1
    gpu.conv3d_device(N, s, d, s, b, flags)
    torch.cuda.synchronize()
    assert torch.equal(s, o)  # in place
    _check(sig, f.astype(np.complex64), o.cpu().numpy(), True)
    assert gpu.device_status() == 0


@pytest.mark.parametrize("at", [0, 2])
def test_filters_in_the_outputs(gpu, at):
    """A filter array that is the output array, and one shared filter inside it: filters count
    as read before any output is written."""
    rng = np.random.default_rng(40 + at)
    sig, f = _c64(rng, (5, N, N, N)), _c64(rng, (5, N, N, N))
    s, o = torch.from_numpy(sig).cuda(), torch.from_numpy(f).cuda()
    if at == 0:
        gpu.conv3d_device(N, s, o, o, 5, gpu.FILTER_PER_SIGNAL)
    else:
        gpu.conv3d_device(N, s, o[at], o, 5, 0)
        f = f[at]
    torch.cuda.synchronize()
    _check(sig, f, o.cpu().numpy(), False)


def test_uneven_graph(gpu):
    rng = np.random.default_rng(50)
    sizes = [16, 32, 16, 16, 64]
    offs = np.cumsum([0] + [n ** 3 for n in sizes])
    jobs = [(n, int(o), int(o), int(o)) for n, o in zip(sizes, offs)]
    for in_place in (False, True):
        sigs, filts = [_c64(rng, (n, n, n)) for n in sizes], [_c64(rng, (n, n, n)) for n in sizes]
        s = torch.from_numpy(np.concatenate([x.ravel() for x in sigs])).cuda()
        f = torch.from_numpy(np.concatenate([x.ravel() for x in filts])).cuda()
        o = s if in_place else torch.empty_like(s)
        gpu.conv3d_uneven_device(jobs, s, f, o, gpu.NORMALIZE)
        torch.cuda.synchronize()
        out = o.cpu().numpy()
        for i, n in enumerate(sizes):
            ref = conv3d(sigs[i], filts[i], "fp32", normalize=True)
            assert snr_db(ref, out[offs[i]:offs[i + 1]].reshape(n, n, n)) > 120.0
