"""Routes of the two-pass transform (twopass.cuh) that share or order their buffers: calls on two
streams, uneven batches whose filters lie among their outputs, and batches in several chunks
whose real filters all go with the first. Tolerance: the reference's criterion, a relative L2
error of 1e-6 against FP64; the same route by another order gives the same bits."""
import numpy as np
import pytest

from oracle import conv3d, rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


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


def _randn(gen, *shape):
    return torch.view_as_complex(torch.randn(shape + (2,), generator=gen, device="cuda"))


@pytest.mark.parametrize("calls", [((128, 5, "shared"), (128, 4, "pairs")), ((256, 3, "shared"), (256, 2, "pairs")),
                                   ((256, 5, "shared"), (128, 9, "spectrum")), ((64, 40, "shared"), (32, 1, "shared")),
                                   ((32, 600, "in_place"), (64, 33, "spectrum")), ((128, 33, "in_place"), (256, 4, "in_place"))])
def test_two_streams(tp, calls):
    """Back to back on two streams, no host wait: as each alone, bit for bit."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(sum(n + b for n, b, _ in calls))
    flags = {"shared": 0, "in_place": 0, "pairs": tp.FILTER_PER_SIGNAL, "spectrum": tp.FILTER_IS_SPECTRUM}
    work = []
    for n, b, how in calls:
        s = _randn(gen, b, n, n, n)
        f = _randn(gen, *((b,) if how == "pairs" else ()), n, n, n)
        work.append((n, b, how, s, f, torch.cuda.Stream()))

    def run(n, b, how, s, f, stream, out):
        tp.conv3d_device(n, out if how == "in_place" else s, f, out, b, flags[how] | tp.NORMALIZE, stream)

    rounds = 3
    outs = [[w[3].clone() for _ in range(rounds)] for w in work]
    alone = [w[3].clone() for w in work]
    torch.cuda.synchronize()
    for w, o in zip(work, alone):
        run(*w, o)
        torch.cuda.synchronize()
    for k in range(rounds):
        for w, o in zip(work, outs):
            run(*w, o[k])
    torch.cuda.synchronize()
    for a, o in zip(alone, outs):
        for k in range(rounds):
            assert torch.equal(a, o[k]), k


@pytest.mark.parametrize("sizes", [[32, 32, 32], [64, 64], [128, 128, 128], [256, 256],
                                   [256, 128, 32, 64, 16, 128, 256, 64, 32, 16]])
def test_uneven_filters_among_the_outputs(tp, sizes):
    """Every job's filter lies in the output of the next job of its size."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(sum(sizes))
    offs = np.cumsum([0] + [n ** 3 for n in sizes])
    classes = {n: [j for j, m in enumerate(sizes) if m == n] for n in sizes}
    at = {}  # the job in whose output j's filter lies
    for js in classes.values():
        at.update({j: js[(i + 1) % len(js)] for i, j in enumerate(js)})
    s, f = _randn(gen, int(offs[-1])), _randn(gen, int(offs[-1]))
    apart, among = torch.empty_like(s), torch.empty_like(s)
    for _ in range(2):  # the second time through cached plans
        for j, n in enumerate(sizes):
            among[offs[at[j]]:offs[at[j]] + n ** 3] = f[offs[j]:offs[j + 1]]
        tp.conv3d_uneven_device([(n, int(o), int(o), int(o)) for n, o in zip(sizes, offs)], s, f, apart, tp.NORMALIZE)
        tp.conv3d_uneven_device([(n, int(offs[j]), int(offs[at[j]]), int(offs[j])) for j, n in enumerate(sizes)],
                                s, among, among, tp.NORMALIZE)
        torch.cuda.synchronize()
        for j, n in enumerate(sizes):
            part = slice(int(offs[j]), int(offs[j + 1]))
            if n != 16:  # those run whole when they can
                assert torch.equal(apart[part], among[part]), (j, n)
            sig, flt, out = (x[part].cpu().numpy().reshape(n, n, n) for x in (s, f, among))
            assert rel_l2(conv3d(sig[None], flt, "fp64", normalize=True, engine="pocketfft")[0], out) < 1e-6
        s.copy_(_randn(gen, int(offs[-1])))


@pytest.mark.parametrize("n,b,edge", [(32, 515, 512), (64, 130, 128), (128, 33, 32), (256, 5, 4)])
def test_chunks_with_real_filters(tp, n, b, edge):
    """In place, through the scratch cubes `edge` at a time; a real filter per signal."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    s, f = _randn(gen, b, n, n, n), torch.randn((b, n, n, n), generator=gen, device="cuda")
    o = s.clone()
    tp.conv3d_device(n, o, f, o, b, tp.FILTER_PER_SIGNAL | tp.FILTER_REAL | tp.NORMALIZE)
    torch.cuda.synchronize()
    for i in {0, edge - 1, edge, b - 1}:
        sig, flt, out = s[i].cpu().numpy(), f[i].cpu().numpy().astype(np.complex64), o[i].cpu().numpy()
        assert rel_l2(conv3d(sig[None], flt, "fp64", normalize=True, engine="pocketfft")[0], out) < 1e-6
