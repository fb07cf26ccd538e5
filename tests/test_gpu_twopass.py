"""The two-pass 3D transform (twopass.cuh; plan kind 4, variant 3, N = 32 to 256).

Every route of it against the oracle: one filter per signal and shared, complex and real,
batches below, at and above the scratch cubes and the shared-filter threshold, in place,
filters in the outputs' memory, and calls it does not take (overlapping or misaligned
operands), which run the three-axis passes. Tolerance: the reference's 120 dB criterion and
a relative L2 error of 1e-6 against FP64 (the FP32 passes are at 3-4e-7).
"""
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


@pytest.fixture
def tp(gpu):
    keep = {(n, k): gpu.plan_variant(n, k) for n in (32, 64, 128, 256) for k in (4, 7)}
    for n in (32, 64, 128, 256):
        assert gpu.plan_variant(n, 4, 3) == 3
        gpu.plan_variant(n, 7, 0)
    gpu.device_status()
    yield gpu
    assert gpu.device_status() == 0
    for (n, k), v in keep.items():
        gpu.plan_variant(n, k, v)


def _check(ref32, ref64, out):
    assert snr_db(ref32, out) > 120.0
    assert rel_l2(ref64, out) < 1e-6


@pytest.mark.parametrize("n,b,filt", [(128, b, f) for b in (1, 2, 3, 4, 7) for f in ("shared", "pairs", "real", "real_pairs")]
                         + [(n, b, f) for n in (32, 64) for b in (2, 5) for f in ("shared", "pairs", "real", "real_pairs")]
                         + [(32, 1100, "shared"), (32, 515, "pairs"), (64, 131, "shared")]
                         + [(256, 1, "real"), (256, 3, "shared"), (256, 5, "shared"), (256, 5, "pairs")])
def test_routes(tp, n, b, filt):
    rng = np.random.default_rng(n + b)
    sig = _c64(rng, (b, n, n, n))
    f = _c64(rng, (b, n, n, n) if filt.endswith("pairs") else (n, n, n))
    flags = (tp.FILTER_PER_SIGNAL if filt.endswith("pairs") else 0) | tp.NORMALIZE
    if filt.startswith("real"):
        f = f.real.copy()
        flags |= tp.FILTER_REAL
    s, d = torch.from_numpy(sig).cuda(), torch.from_numpy(f).cuda()
    o = torch.empty_like(s)
    tp.conv3d_device(n, s, d, o, b, flags)
    tp.conv3d_device(n, s, d, s, b, flags)  # in place, through the scratch cubes
    torch.cuda.synchronize()
    out, inplace = o.cpu().numpy(), s.cpu().numpy()
    some = range(b) if n == 128 else (0, b - 1)
    for i in some:
        fi = (f[i] if filt.endswith("pairs") else f).astype(np.complex64)
        ref = conv3d(sig[i:i + 1], fi, "fp32", normalize=True, engine="pocketfft")[0]
        ref64 = conv3d(sig[i:i + 1], fi, "fp64", normalize=True, engine="pocketfft")[0]
        _check(ref, ref64, out[i])
        _check(ref, ref64, inplace[i])


@pytest.mark.parametrize("n,b,off", [(32, 2, 0), (32, 515, 1), (64, 1, 0), (64, 5, 1), (64, 9, 0), (128, 1, 1),
                                     (128, 33, 0), (256, 1, 0), (256, 4, 1)])
def test_given_spectrum(tp, n, b, off):
    """Signals against a spectrum in natural order, at 16- and 8-byte alignment, apart and in place."""
    rng = np.random.default_rng(n + b)
    sig, f = _c64(rng, (b, n, n, n)), _c64(rng, (n, n, n))
    spec = torch.empty(n ** 3 + off, dtype=torch.complex64, device="cuda")[off:]
    spec.copy_(torch.from_numpy(np.fft.fftn(f.astype(np.complex128)).astype(np.complex64)).flatten())
    s = torch.from_numpy(sig).cuda()
    o = torch.empty_like(s)
    flags = tp.FILTER_IS_SPECTRUM | tp.NORMALIZE
    tp.conv3d_device(n, s, spec, o, b, flags)
    tp.conv3d_device(n, s, spec, s, b, flags)
    torch.cuda.synchronize()
    assert torch.equal(o, s)
    for i in {0, b // 2, b - 1}:
        _check(conv3d(sig[i:i + 1], f, "fp32", normalize=True, engine="pocketfft")[0],
               conv3d(sig[i:i + 1], f, "fp64", normalize=True, engine="pocketfft")[0], o[i].cpu().numpy())


def test_filters_in_the_outputs(tp):
    """The filters are read before any output is written, chunk by chunk or not."""
    n, b = 128, 5
    rng = np.random.default_rng(7)
    sig, f = _c64(rng, (b, n, n, n)), _c64(rng, (b, n, n, n))
    s, o = torch.from_numpy(sig).cuda(), torch.from_numpy(f).cuda()
    apart = torch.empty_like(s)
    tp.conv3d_device(n, s, o, apart, b, tp.FILTER_PER_SIGNAL)
    tp.conv3d_device(n, s, o, o, b, tp.FILTER_PER_SIGNAL)
    torch.cuda.synchronize()
    assert torch.equal(o, apart)
    _check(conv3d(sig[4:], f[4], "fp32", engine="pocketfft")[0], conv3d(sig[4:], f[4], "fp64", engine="pocketfft")[0],
           o[4].cpu().numpy())


def test_operands_it_does_not_take(tp):
    """8-byte aligned operands run the three-axis passes, with the same results."""
    n, b = 128, 2
    rng = np.random.default_rng(8)
    sig, f = _c64(rng, (b, n, n, n)), _c64(rng, (n, n, n))
    ref = conv3d(sig, f, "fp32", engine="pocketfft")
    v = n ** 3
    for which in range(3):
        bufs = [torch.empty(k * v + 1, dtype=torch.complex64, device="cuda") for k in (b, 1, b)]
        s, d, o = (x[(1 if i == which else 0):][:x.numel() - 1] for i, x in enumerate(bufs))
        s.copy_(torch.from_numpy(sig).flatten())
        d.copy_(torch.from_numpy(f).flatten())
        tp.conv3d_device(n, s, d, o, b, 0)
        torch.cuda.synchronize()
        assert snr_db(ref, o.cpu().numpy().reshape(sig.shape)) > 120.0, which


@pytest.mark.parametrize("in_place", [False, True])
def test_uneven_graph(tp, in_place):
    """The graph's classes run it in table mode unless a job of the class is in place; the
    cached plan follows the buffers either way."""
    sizes = [256, 128, 32, 64, 128, 64, 256, 32, 128]
    offs = np.cumsum([0] + [n ** 3 for n in sizes])
    jobs = [(n, int(o), int(o), int(o)) for n, o in zip(sizes, offs)]
    for rep in range(2):
        rng = np.random.default_rng(90 + rep)
        sigs, filts = [_c64(rng, (n, n, n)) for n in sizes], [_c64(rng, (n, n, n)) for n in sizes]
        s = torch.from_numpy(np.concatenate([x.ravel() for x in sigs])).cuda()
        f = torch.from_numpy(np.concatenate([x.ravel() for x in filts])).cuda()
        o = s if in_place else torch.empty_like(s)
        tp.conv3d_uneven_device(jobs, s, f, o, tp.NORMALIZE)
        torch.cuda.synchronize()
        out = o.cpu().numpy()
        for i, n in enumerate(sizes):
            ref = conv3d(sigs[i], filts[i], "fp32", normalize=True, engine="pocketfft")
            assert snr_db(ref, out[offs[i]:offs[i + 1]].reshape(n, n, n)) > 120.0, (rep, i, n)


def test_captured_call(tp):
    """A call captured into a graph after a first one replays on new data."""
    n, b = 128, 4
    rng = np.random.default_rng(9)
    sig, f = _c64(rng, (b, n, n, n)), _c64(rng, (n, n, n))
    s, d = torch.from_numpy(sig).cuda(), torch.from_numpy(f).cuda()
    o = torch.empty_like(s)
    tp.conv3d_device(n, s, d, o, b, 0)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        tp.conv3d_device(n, s, d, o, b, 0, torch.cuda.current_stream())
    sig2 = _c64(rng, (b, n, n, n))
    s.copy_(torch.from_numpy(sig2))
    g.replay()
    torch.cuda.synchronize()
    assert snr_db(conv3d(sig2, f, "fp32", engine="pocketfft"), o.cpu().numpy()) > 120.0


def test_alternating_with_the_staged_pass(tp):
    """Calls that run the L2-staged pass between calls that run the two-pass transform, on
    the same buffers and without waiting in between."""
    n, b = 128, 4
    rng = np.random.default_rng(10)
    sig, f = _c64(rng, (b, n, n, n)), _c64(rng, (b, n, n, n))
    s, d = torch.from_numpy(sig).cuda(), torch.from_numpy(f).cuda()
    o, spec = torch.empty_like(s), torch.empty_like(s)
    for _ in range(20):
        tp.filter_spectrum_device(n, d, spec, b)
        tp.conv3d_device(n, s, d, o, b, tp.FILTER_PER_SIGNAL)
    torch.cuda.synchronize()
    i = b - 1
    assert snr_db(conv3d(sig[i:], f[i], "fp32", engine="pocketfft")[0], o[i].cpu().numpy()) > 120.0
    assert rel_l2(np.fft.fftn(f[i].astype(np.complex128)), spec[i].cpu().numpy()) < 1e-6
