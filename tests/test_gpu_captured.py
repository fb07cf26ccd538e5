"""Calls captured into a graph, and what their replays leave behind.

A replay uses the counters that the capture recorded, so a launch that gave up, or other
launches in between, must leave nothing in them. Expected values are those of the same call
made directly, bit for bit.
"""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

STATUS_QUEUE = 2  # a grid barrier gave up


def _cubes(gen, *shape):
    return torch.view_as_complex(torch.randn(shape + (2,), generator=gen, device="cuda"))


def _capture(call):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call(torch.cuda.current_stream())
    return g


@pytest.fixture
def cg(gpu):
    gpu.device_status()
    yield gpu
    gpu.debug_dependency_wait_limit(-1)
    gpu.device_status()


@pytest.mark.parametrize("n", [32, 64])
def test_replays_of_one_small_cube_after_one_that_gave_up(cg, n):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    s, f = _cubes(gen, n, n, n), _cubes(gen, n, n, n)
    out, want = torch.empty_like(s), torch.empty_like(s)
    cg.conv3d_device(n, s, f, want, 1, 0)  # scratch is allocated outside the capture
    torch.cuda.synchronize()
    g = _capture(lambda stream: cg.conv3d_device(n, s, f, out, 1, 0, stream))
    cg.debug_dependency_wait_limit(0)
    g.replay()
    assert cg.device_status() & STATUS_QUEUE
    cg.debug_dependency_wait_limit(-1)

    def replay():
        s.copy_(_cubes(gen, n, n, n))
        f.copy_(_cubes(gen, n, n, n))
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        cg.conv3d_device(n, s, f, want, 1, 0)
        torch.cuda.synchronize()
        assert cg.device_status() == 0
        assert torch.equal(out, want)

    for _ in range(4):
        replay()
    # direct launches in between, some of which give up
    cg.debug_dependency_wait_limit(0)
    for _ in range(3):
        cg.conv3d_device(n, s, f, want, 1, 0)
    assert cg.device_status() & STATUS_QUEUE
    cg.debug_dependency_wait_limit(-1)
    for _ in range(40):
        cg.conv3d_device(n, s, f, want, 1, 0)
    for _ in range(4):
        replay()


@pytest.mark.parametrize("n", [32, 64, 128, 256])
@pytest.mark.parametrize("what", ["spectrum", "conv"])
def test_a_first_call_of_its_size_captured_without_a_workspace(cg, n, what):
    """A spectrum, or a convolution with one, needs no workspace: with the default plan it can be
    captured before any call of its size has allocated what faster routes use."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    keep = cg.plan_variant(n, 4)
    cg.fpga_final()
    assert cg.fpga_initialize("cuda:0", "convgpu_plans.json", False) == 0
    try:
        src, f, out, want = (_cubes(gen, n, n, n) for _ in range(4))

        def call(dst, stream=None):
            if what == "spectrum":
                cg.filter_spectrum_device(n, src, dst, 1, stream)
            else:
                cg.conv3d_device(n, src, f, dst, 1, cg.FILTER_IS_SPECTRUM, stream)

        cg.plan_variant(n, 4, 0)  # separate passes: nothing is allocated
        call(want)
        torch.cuda.synchronize()
        assert cg.plan_variant(n, 4, 3) == 3
        g = _capture(lambda stream: call(out, stream))
        for _ in range(2):
            src.copy_(_cubes(gen, n, n, n))
            out.zero_()
            g.replay()
            torch.cuda.synchronize()
            cg.plan_variant(n, 4, 0)
            call(want)
            torch.cuda.synchronize()
            assert torch.equal(out, want)
        assert cg.device_status() == 0
    finally:
        cg.plan_variant(n, 4, keep)
