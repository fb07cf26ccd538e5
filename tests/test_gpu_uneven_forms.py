"""Forms of an uneven batch's size classes (grouped.cu): tiles (3 launches) or axis passes (7), by
the number of jobs and the classes beside; 16^3 jobs run whole (1). Sizes on either side of
every line, apart and in place (always by axis passes here). The launches are counted, and
every job is compared with its own call (2e-6: two results of 1e-6 each against FP64, the
criterion of the FP32 passes)."""
import numpy as np
import pytest

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


@pytest.mark.parametrize("jobs,launches", [
    ({32: 1}, 3), ({32: 20}, 3), ({32: 21}, 7), ({32: 169}, 7), ({32: 170}, 3), ({32: 20, 16: 3}, 4),
    ({64: 1}, 3), ({64: 13}, 3), ({64: 2, 32: 2}, 6), ({64: 2, 32: 3}, 14), ({64: 13, 32: 5}, 14), ({64: 14, 32: 5}, 10),
    ({128: 1}, 3), ({128: 1, 64: 1, 32: 9}, 17), ({128: 1, 64: 2, 32: 1}, 21), ({128: 1, 64: 7}, 14), ({128: 1, 64: 8}, 6),
    ({128: 1, 64: 14, 32: 33}, 13), ({128: 1, 32: 31}, 10), ({128: 1, 32: 32}, 14), ({128: 2, 64: 4, 32: 1}, 17),
    ({128: 2, 64: 8, 16: 2}, 7), ({256: 1, 128: 1, 64: 3, 32: 2, 16: 1}, 25)])
def test_classes(tp, jobs, launches):
    sizes = [n for n, k in jobs.items() for _ in range(k)]
    order = np.random.default_rng(len(sizes)).permutation(len(sizes))
    sizes = [sizes[i] for i in order]
    offs = np.cumsum([0] + [n ** 3 for n in sizes])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(len(sizes))
    s = torch.view_as_complex(torch.randn((int(offs[-1]), 2), generator=gen, device="cuda"))
    f = torch.view_as_complex(torch.randn((int(offs[-1]), 2), generator=gen, device="cuda"))
    o, inplace = torch.empty_like(s), s.clone()
    batch = [(n, int(at), int(at), int(at)) for n, at in zip(sizes, offs)]
    before = tp.launch_count()
    tp.conv3d_uneven_device(batch, s, f, o, tp.NORMALIZE)
    assert tp.launch_count() - before == launches
    tp.conv3d_uneven_device(batch, inplace, f, inplace, tp.NORMALIZE)
    torch.cuda.synchronize()
    for n, at in zip(sizes, offs):
        part = slice(int(at), int(at) + n ** 3)
        want = torch.empty_like(s[part])
        tp.conv3d_device(n, s[part], f[part], want, 1, tp.NORMALIZE)
        scale = float(torch.linalg.vector_norm(want))
        for got in (o[part], inplace[part]):
            assert float(torch.linalg.vector_norm(got - want)) < 2e-6 * scale, n
