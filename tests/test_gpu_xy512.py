"""The L2-staged x+y pass of N = 512 on pairs (xy512.cuh) against the separate passes, forward
and inverse, on one and two cubes, in place; and its dependency waits giving up.

Both routes are within the 3-4e-7 of the FP32 passes, so 1e-6 apart at most."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
N, XY = 512, 4


@pytest.mark.parametrize("b", [1, 2])
def test_against_separate_passes(gpu, b):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(b)
    x = torch.view_as_complex(torch.randn((b, N, N, N, 2), generator=gen, device="cuda"))
    f = torch.view_as_complex(torch.randn((N, N, N, 2), generator=gen, device="cuda"))
    keep = gpu.plan_variant(N, XY)
    gpu.device_status()
    spec, outs = [], []
    for v in (0, 1):
        assert gpu.plan_variant(N, XY, v) == v
        s = torch.empty_like(x)
        gpu.filter_spectrum_device(N, x, s, b)
        spec.append(s)
        o = x.clone()
        gpu.conv3d_device(N, o, f, o, b, gpu.NORMALIZE)
        outs.append(o)
    torch.cuda.synchronize()
    gpu.plan_variant(N, XY, keep)
    assert gpu.device_status() == 0
    for a, c in (spec, outs):
        assert float(torch.linalg.vector_norm(a - c) / torch.linalg.vector_norm(a)) < 1e-6
        assert not torch.equal(a, c)


def test_dependency_waits_that_give_up_are_reported(gpu):
    x = torch.ones((N, N, N), dtype=torch.complex64, device="cuda")
    s = torch.empty_like(x)
    keep = gpu.plan_variant(N, XY)
    gpu.plan_variant(N, XY, 1)
    try:
        gpu.device_status()
        gpu.debug_dependency_wait_limit(0)
        gpu.filter_spectrum_device(N, x, s, 1)
        torch.cuda.synchronize()
        assert gpu.device_status() == 16
        gpu.debug_dependency_wait_limit(-1)
        gpu.filter_spectrum_device(N, x, s, 1)
        torch.cuda.synchronize()
        assert gpu.device_status() == 0
        assert abs(s[0, 0, 0].item() - N ** 3) < 1 and float(s.flatten()[1:].abs().max()) < 1
    finally:
        gpu.debug_dependency_wait_limit(-1)
        gpu.plan_variant(N, XY, keep)
