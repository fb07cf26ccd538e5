"""The autotuner at N = 512: it times what its choice decides. The fused z pass of the calls in the
library's order is one kernel, so kind 3 keeps variant 0; kind 2 is for the unordered calls."""
import pytest

pytestmark = [pytest.mark.gpu, pytest.mark.slow]
torch = pytest.importorskip("torch")
N, KINDS = 512, 8


def test_choices_and_calls(gpu):
    keep = [gpu.plan_variant(N, k) for k in range(KINDS)]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(N)
    try:
        gpu.plan_variant(N, 3, 1)
        gpu.autotune([N], write_cache=False)
        assert gpu.plan_variant(N, 3) == 0
        chosen = gpu.plan_variant(N, 2)
        s = torch.view_as_complex(torch.randn((N, N, N, 2), generator=gen, device="cuda"))
        f = torch.view_as_complex(torch.randn((N, N, N, 2), generator=gen, device="cuda"))
        spec, outs = torch.empty_like(f), []
        gpu.filter_spectrum_device(N, f, spec, 1)
        for call, variants in ((gpu.conv3d_device, (0, 1)), (gpu.conv3d_device_noalloc, (chosen, 1 - chosen))):
            for v in variants:
                gpu.plan_variant(N, 2, v)
                gpu.plan_variant(N, 3, v)
                o = torch.empty_like(s)
                call(N, s, spec, o, 1, gpu.FILTER_IS_SPECTRUM | gpu.NORMALIZE)
                outs.append(o)
            o = torch.empty_like(s)
        gpu.plan_variant(N, 3, 1)
        gpu.conv3d_device(N, s, f, o, 1, gpu.NORMALIZE)  # the filter's z transform in the z pass
        outs.append(o)
        torch.cuda.synchronize()
        assert torch.equal(outs[0], outs[1])
        for o in outs[1:]:  # two results of 1e-6 each
            assert float(torch.linalg.vector_norm(o - outs[0]) / torch.linalg.vector_norm(outs[0])) < 2e-6
        assert gpu.device_status() == 0
    finally:
        for k, v in enumerate(keep):
            gpu.plan_variant(N, k, v)
