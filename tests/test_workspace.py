"""The workspace a call asks for holds what the call writes to it, by the route it takes."""
import pytest

import convfpga_gb300 as cg

HERM = 7  # plan kind: half spectra of real filters


@pytest.mark.parametrize("n", [16, 32, 64])
@pytest.mark.parametrize("per_signal", [0, cg.FILTER_PER_SIGNAL])
def test_one_small_cube_with_a_real_filter(built_lib, n, per_signal):
    """One launch does it (N <= 64, one cube), with the filter's N^3 values in the workspace, whatever
    the plan says of half spectra, which the launch does not use."""
    keep = cg.plan_variant(n, HERM)
    try:
        for herm in (0, 1):
            cg.plan_variant(n, HERM, herm)
            assert cg.workspace_bytes(n, 1, cg.FILTER_REAL | per_signal) >= n ** 3 * 8
    finally:
        cg.plan_variant(n, HERM, keep)


@pytest.mark.gpu
def test_one_small_cube_with_a_real_filter_in_a_new_workspace(gpu):
    import numpy as np
    import torch
    from oracle import conv3d, rel_l2

    n = 64
    rng = np.random.default_rng(64)
    sig = (rng.uniform(-1, 1, (1, n, n, n)) + 1j * rng.uniform(-1, 1, (1, n, n, n))).astype(np.complex64)
    filt = rng.uniform(-1, 1, (n, n, n)).astype(np.float32)
    gpu.fpga_final()
    assert gpu.fpga_initialize("cuda:0", "convgpu_plans.json", False) == 0
    keep = gpu.plan_variant(n, HERM)
    gpu.plan_variant(n, HERM, 1)
    s = torch.from_numpy(sig).cuda()
    gpu.conv3d_device(n, s, torch.from_numpy(filt).cuda(), s, 1, gpu.FILTER_REAL)
    torch.cuda.synchronize()
    gpu.plan_variant(n, HERM, keep)
    assert gpu.device_status() == 0
    assert rel_l2(conv3d(sig, filt.astype(np.complex64), "fp64", engine="pocketfft"), s.cpu().numpy()) < 1e-6
