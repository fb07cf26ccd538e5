"""Calls that overlap on the GPU.

The no-allocation entry point is not ordered with any other call; with a given spectrum it
uses no scratch, so it may run beside any call, at N = 512 too, where the fused z pass of the
regular entry points takes its tiles from a counter that launches share.
"""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [128, 512])
@pytest.mark.parametrize("beside", ["conv3d_device", "conv3d_device_noalloc"])
def test_noalloc_with_a_spectrum_beside_other_calls(gpu, n, beside):
    """Two streams, no waits between them: each result is that of its call made alone, bit for bit."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)

    def cube():
        return torch.view_as_complex(torch.randn((n, n, n, 2), generator=gen, device="cuda"))

    sig, filt = [cube(), cube()], [cube(), cube()]
    spec = [torch.empty_like(f) for f in filt]
    for f, s in zip(filt, spec):
        gpu.filter_spectrum_device(n, f, s, 1)
    calls = [gpu.conv3d_device_noalloc, getattr(gpu, beside)]
    alone, out = [torch.empty_like(s) for s in sig], [torch.empty_like(s) for s in sig]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    gpu.device_status()
    torch.cuda.synchronize()
    for k in range(2):
        calls[k](n, sig[k], spec[k], alone[k], 1, gpu.FILTER_IS_SPECTRUM | gpu.NORMALIZE, streams[k])
        torch.cuda.synchronize()
    for _ in range(4):
        for k in range(2):
            calls[k](n, sig[k], spec[k], out[k], 1, gpu.FILTER_IS_SPECTRUM | gpu.NORMALIZE, streams[k])
    torch.cuda.synchronize()
    assert gpu.device_status() == 0
    for k in range(2):
        assert torch.equal(alone[k], out[k]), k
    # each spectrum's own filter: convolved with an impulse it comes back
    s = torch.zeros_like(sig[0])
    s[0, 0, 0] = 1
    calls[0](n, s, spec[0], s, 1, gpu.FILTER_IS_SPECTRUM | gpu.NORMALIZE, streams[0])
    torch.cuda.synchronize()
    assert float(torch.linalg.vector_norm(s - filt[0]) / torch.linalg.vector_norm(filt[0])) < 1e-6


@pytest.mark.parametrize("n,b", [(32, 2), (64, 1), (64, 33), (128, 1), (128, 8), (256, 3)])
def test_spectrum_written_just_before_it_is_used(gpu, n, b):
    """filter_spectrum_device, then the convolution with that spectrum, on a new filter each time
    and with no wait between: as with a wait, bit for bit."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n + b)
    keep = gpu.plan_variant(n, 4)
    gpu.plan_variant(n, 4, 3)

    def cubes(k):
        return torch.view_as_complex(torch.randn((k, n, n, n, 2), generator=gen, device="cuda"))

    sig, filts = cubes(b), cubes(6)
    spec, flags = torch.empty_like(filts[0]), gpu.FILTER_IS_SPECTRUM | gpu.NORMALIZE
    outs, want = [torch.empty_like(sig) for _ in filts], torch.empty_like(sig)
    gpu.device_status()
    gpu.conv3d_device(n, sig, filts[0], want, b, flags)  # any allocation happens here
    torch.cuda.synchronize()
    for f, o in zip(filts, outs):
        gpu.filter_spectrum_device(n, f, spec, 1)
        gpu.conv3d_device(n, sig, spec, o, b, flags)
    torch.cuda.synchronize()
    for f, o in zip(filts, outs):
        gpu.filter_spectrum_device(n, f, spec, 1)
        torch.cuda.synchronize()
        gpu.conv3d_device(n, sig, spec, want, b, flags)
        torch.cuda.synchronize()
        assert torch.equal(o, want)
    gpu.plan_variant(n, 4, keep)
    assert gpu.device_status() == 0
