"""Calls whose scratch cannot be allocated run the routes that need none, this time and the
next, until fpga_final. Allocations are failed on the host through the library's testing hook.
Tolerance: the reference's criterion, a relative L2 error of 1e-6 against FP64."""
import numpy as np
import pytest

from oracle import conv3d, rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

XY = 4


def _c64(rng, shape):
    return (rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape)).astype(np.complex64)


def _renew(cg):
    cg.fpga_final()
    assert cg.fpga_initialize("cuda:0", "convgpu_plans.json", False) == 0


@pytest.fixture
def fresh(gpu):
    """Nothing allocated, the default plans."""
    keep = {(n, k): gpu.plan_variant(n, k) for n in (32, 64, 128, 256) for k in (XY, 7)}
    _renew(gpu)
    for n in (32, 64, 128, 256):
        gpu.plan_variant(n, XY, 3)
        gpu.plan_variant(n, 7, 0)
    gpu.device_status()
    yield gpu
    gpu.debug_fail_allocations(0)
    for (n, k), v in keep.items():
        gpu.plan_variant(n, k, v)
    _renew(gpu)


def _launches(cg, call):
    before = cg.launch_count()
    call()
    torch.cuda.synchronize()
    assert cg.device_status() == 0
    return cg.launch_count() - before


@pytest.mark.parametrize("n,b", [(32, 5), (64, 3), (128, 3), (256, 2)])
@pytest.mark.parametrize("filt", ["shared", "spectrum", "pairs_in_place"])
def test_batches(fresh, n, b, filt):
    cg, rng = fresh, np.random.default_rng(n)
    pairs = filt == "pairs_in_place"
    sig, f = _c64(rng, (b, n, n, n)), _c64(rng, (b, n, n, n) if pairs else (n, n, n))
    flags = (cg.FILTER_PER_SIGNAL if pairs else cg.FILTER_IS_SPECTRUM if filt == "spectrum" else 0) | cg.NORMALIZE
    d = f if filt != "spectrum" else np.fft.fftn(f.astype(np.complex128)).astype(np.complex64)
    s0, d = torch.from_numpy(sig).cuda(), torch.from_numpy(d).cuda()
    refs = [conv3d(sig[i:i + 1], f[i] if pairs else f, "fp64", normalize=True, engine="pocketfft")[0] for i in (0, b - 1)]

    def run():
        s = s0.clone()
        o = s if pairs else torch.empty_like(s)
        count = _launches(cg, lambda: cg.conv3d_device(n, s, d, o, b, flags))
        for i, ref in zip((0, b - 1), refs):
            assert rel_l2(ref, o[i].cpu().numpy()) < 1e-6
        return count

    cg.plan_variant(n, XY, 0)
    separate = run()  # allocates the workspace
    cg.plan_variant(n, XY, 3)
    cg.debug_fail_allocations(2 if n >= 128 else 1)  # the scratch cubes and the staged pass's ring
    assert run() == separate
    assert run() == separate
    cg.debug_fail_allocations(0)
    _renew(cg)
    # three spectrum calls of 128^3 lie between the batches that run in tiles: as many launches
    assert run() < separate or (n, filt) == (128, "spectrum")


@pytest.mark.parametrize("n", [32, 64])
@pytest.mark.parametrize("real", [False, True])
def test_one_small_cube(fresh, n, real):
    """Whole planes and z tiles instead of tiles (k_small_conv), directly and captured, also after
    a launch that gave up."""
    cg, rng = fresh, np.random.default_rng(n)
    sig, f = _c64(rng, (n, n, n)), _c64(rng, (n, n, n))
    if real:
        f = f.real.copy()
    flags = cg.FILTER_REAL if real else 0
    s, d = torch.from_numpy(sig).cuda(), torch.from_numpy(f).cuda()
    o = torch.empty_like(s)
    ref = conv3d(sig[None], f.astype(np.complex64), "fp64", engine="pocketfft")[0]
    two = torch.from_numpy(_c64(rng, (2, n, n, n))).cuda()
    cg.plan_variant(n, XY, 0)
    cg.conv3d_device(n, two, d, two, 2, flags)  # allocates the workspace
    cg.plan_variant(n, XY, 3)
    cg.debug_fail_allocations(1)
    for _ in range(2):
        o.zero_()
        assert _launches(cg, lambda: cg.conv3d_device(n, s, d, o, 1, flags)) == 1
        assert rel_l2(ref, o.cpu().numpy()) < 1e-6
    direct = o.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        cg.conv3d_device(n, s, d, o, 1, flags, torch.cuda.current_stream())
    cg.debug_dependency_wait_limit(0)
    g.replay()
    assert cg.device_status() & 2
    cg.debug_dependency_wait_limit(-1)
    for k in (2, 1, 2):
        s.copy_(torch.from_numpy(k * sig))
        g.replay()
        torch.cuda.synchronize()
        assert cg.device_status() == 0
        assert torch.equal(o, k * direct)


@pytest.mark.parametrize("n", [128, 256])
def test_uneven_in_place_without_the_ring(fresh, n):
    """Two jobs: one of 128^3 would not ask for it."""
    cg, rng = fresh, np.random.default_rng(n)
    sig, f = _c64(rng, (2, n, n, n)), _c64(rng, (2, n, n, n))
    s, d = torch.from_numpy(sig).cuda(), torch.from_numpy(f).cuda()
    cg.debug_fail_allocations(1)
    cg.conv3d_uneven_device([(n, i * n ** 3, i * n ** 3, i * n ** 3) for i in range(2)], s, d, s, cg.NORMALIZE)
    torch.cuda.synchronize()
    assert cg.device_status() == 0
    for i in range(2):
        ref = conv3d(sig[i:i + 1], f[i], "fp64", normalize=True, engine="pocketfft")[0]
        assert rel_l2(ref, s[i].cpu().numpy()) < 1e-6


@pytest.mark.parametrize("n,b", [(32, 3), (64, 2), (128, 2), (256, 1)])
def test_calls_that_need_no_scratch_ask_for_none(fresh, n, b):
    """A filter per signal, outputs apart: the failure waits for the first call in place."""
    cg, rng = fresh, np.random.default_rng(n)
    sig, f = _c64(rng, (b, n, n, n)), _c64(rng, (b, n, n, n))
    s, d = torch.from_numpy(sig).cuda(), torch.from_numpy(f).cuda()
    o = torch.empty_like(s)
    cg.plan_variant(n, XY, 0)
    cg.conv3d_device(n, s, d, o, b, cg.FILTER_PER_SIGNAL)  # allocates the workspace
    torch.cuda.synchronize()
    cg.plan_variant(n, XY, 3)
    cg.debug_fail_allocations(2 if n >= 128 else 1)
    assert _launches(cg, lambda: cg.conv3d_device(n, s, d, o, b, cg.FILTER_PER_SIGNAL)) == 3
    assert rel_l2(conv3d(sig[:1], f[0], "fp64", engine="pocketfft")[0], o[0].cpu().numpy()) < 1e-6
    assert _launches(cg, lambda: cg.conv3d_device(n, s, d, s, b, cg.FILTER_PER_SIGNAL)) > 3
    assert rel_l2(conv3d(sig[:1], f[0], "fp64", engine="pocketfft")[0], s[0].cpu().numpy()) < 1e-6


def test_scratch_makes_room_for_what_a_call_needs(fresh):
    """A workspace that finds no memory takes that of the scratch cubes; later calls do without
    them. Scratch cubes that a captured call holds stay."""
    cg, n = fresh, 128
    rng = np.random.default_rng(n)
    sig, f = _c64(rng, (5, n, n, n)), _c64(rng, (5, n, n, n))
    s, d = torch.from_numpy(sig).cuda(), torch.from_numpy(f).cuda()
    o = torch.empty_like(s)

    def shared(stream=None):
        cg.conv3d_device(n, s, d, o, 3, 0, stream)  # through the scratch cubes; one filter of workspace

    def check(i, fi):
        assert rel_l2(conv3d(sig[i:i + 1], f[fi], "fp64", engine="pocketfft")[0], o[i].cpu().numpy()) < 1e-6

    assert _launches(cg, shared) == 3
    check(2, 0)
    cg.debug_fail_allocations(1)
    cg.conv3d_device(n, s, d, o, 5, cg.FILTER_PER_SIGNAL)  # five filters of workspace
    torch.cuda.synchronize()
    check(4, 4)
    assert _launches(cg, shared) > 3
    check(2, 0)
    _renew(cg)
    assert _launches(cg, shared) == 3
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        shared(torch.cuda.current_stream())
    o.zero_()
    g.replay()
    torch.cuda.synchronize()
    check(2, 0)
    cg.debug_fail_allocations(1)
    with pytest.raises(cg.ConvGpuError):
        cg.conv3d_device(n, s, d, o, 5, cg.FILTER_PER_SIGNAL)
    assert _launches(cg, shared) == 3
    check(2, 0)
