"""The convolutions that a user of this framework runs, as timed cases.

Sizes and distributions are those of the framework's own workloads (bench.py) and the
sizes around them: cubes of 16..512 points a side, one filter for the whole batch, one per
signal, real filters, precomputed spectra, uneven batches, host buffers and the
tensor-core split path. Every case runs with the autotuned plan of its sizes, which a
program makes once and keeps.
"""
import math

import numpy as np
import torch

import convfpga_gb300 as cg

SIZES = (16, 32, 64, 128, 256, 512)
_tuned = set()


def listed():
    return [
        # The smallest call there is: one 16^3 cube, bound by latency.
        _conv("n16_single", 16, 1, filt="shared", normalize=True),
        # bench.py's 64^3 workload: one cube, one complex filter, normalised.
        _conv("n64_single", 64, 1, filt="shared", normalize=True),
        # Many small fields under one kernel (template matching, patches): 100 cubes of 32^3.
        _conv("n32_batch100", 32, 100, filt="shared"),
        # A filter transformed once and used again and again: 33 cubes of 64^3 against its spectrum.
        _conv("n64_spectrum33", 64, 33, filt="spectrum", normalize=True),
        # bench.py's 128^3 workload: 8 signals smoothed by one real Gaussian.
        _conv("n128_batch8_real", 128, 8, filt="real", normalize=False),
        # What a program written for the reference calls: pageable host buffers, one complex filter.
        {"name": "n128_batch8_host", "kind": "host", "n": 128, "batch": 8},
        # bench.py's headline workload: 4 pairs of 256^3 signals and filters ...
        _conv("n256_pairs4", 256, 4, filt="pairs"),
        # ... and the same on the tensor-core split path.
        _conv("n256_pairs4_split", 256, 4, filt="pairs", split=True),
        # An odd batch of large cubes under one complex filter (simulation fields).
        _conv("n256_shared3", 256, 3, filt="shared", normalize=True),
        # The transform of two large filters, kept for later calls.
        {"name": "n256_transform2", "kind": "transform", "n": 256, "batch": 2},
        # bench.py's 512^3 workload: one large field smoothed by a real Gaussian.
        _conv("n512_real", 512, 1, filt="real", normalize=False),
        # bench.py's uneven workload: 96 jobs of 32..256 points a side, a Gaussian filter each.
        {"name": "uneven96", "kind": "uneven", "jobs": 96, "points": 1 << 29, "sizes_seed": 4, "smallest": 32},
    ]


def draw(rng):
    """One more case: the entry point by how often it is used, sizes and batches over their whole range."""
    kind = rng.choice(("conv", "conv", "conv", "conv", "conv", "split", "uneven", "host", "transform"))
    if kind == "uneven":
        return {"kind": "uneven", "jobs": int(round(2 ** rng.uniform(1, 6.5))), "points": 1 << rng.randint(23, 26),
                "sizes_seed": rng.randrange(1 << 20), "smallest": rng.choice((16, 32))}
    if kind == "host":
        n = rng.choice((32, 64, 128))
        return {"kind": "host", "n": n, "batch": _batch(rng, n, 1 << 24)}
    if kind == "transform":
        n = rng.choice(SIZES[:5])
        return {"kind": "transform", "n": n, "batch": _batch(rng, n, 1 << 25)}
    if kind == "split":
        return _conv(None, 256, rng.randint(1, 4), filt=rng.choice(("shared", "pairs")), normalize=rng.random() < 0.5, split=True)
    n = rng.choice(SIZES)
    if n == 512:
        return _conv(None, n, 1, filt=rng.choice(("shared", "real", "spectrum")), normalize=rng.random() < 0.5)
    return _conv(None, n, _batch(rng, n, 1 << 26), filt=rng.choice(("shared", "shared", "pairs", "real", "spectrum")),
                 normalize=rng.random() < 0.5)


def _conv(name, n, batch, filt, normalize=False, split=False):
    case = {"kind": "conv", "n": n, "batch": batch, "filter": filt, "normalize": normalize, "split": split}
    return {"name": name, **case} if name else case


def _batch(rng, n, points):
    """Spread over the logarithm, at most `points` points and 1000 cubes in all."""
    return int(2 ** rng.uniform(0, math.log2(min(1000, max(1, points // n ** 3)) + 0.99)))


def _sizes(case):
    """Job sizes of an uneven batch: {32, 64, 128, 256} with probabilities {.4, .3, .2, .1}
    (with 16 in front: halved for it), at most `points` points together."""
    rng = np.random.default_rng(case["sizes_seed"])
    sizes, p = ([32, 64, 128, 256], [0.4, 0.3, 0.2, 0.1])
    if case["smallest"] == 16:
        sizes, p = [16] + sizes, [0.2, 0.2] + p[1:]
    got, left = [], case["points"]
    for n in rng.choice(sizes, size=case["jobs"], p=p):
        n = int(n)
        while n ** 3 > left and n > case["smallest"]:
            n //= 2
        got.append(n)
        left = max(0, left - n ** 3)
    return got


def _complex(gen, shape, normal=False):
    """complex64 on the GPU: re and im uniform in [-1, 1], or standard normal."""
    x = torch.empty(tuple(shape) + (2,), dtype=torch.float32, device="cuda")
    x.normal_(generator=gen) if normal else x.uniform_(-1, 1, generator=gen)
    return torch.view_as_complex(x)


def _gaussian(n, sigma):
    """Real isotropic Gaussian of unit sum, centred at the origin with periodic wrap."""
    d = torch.arange(n, dtype=torch.float64, device="cuda")
    d = torch.minimum(d, n - d)
    g = torch.exp(-0.5 * (d / sigma) ** 2)
    g = g / g.sum()
    return (g[:, None, None] * g[None, :, None] * g[None, None, :]).float()


def _blobs(gen, n):
    """A smooth field: 64 Gaussian blobs of widths 4..32 points and amplitudes in [-1, 1], with noise of 1e-3."""
    u = torch.rand(64, 5, dtype=torch.float32, device="cuda", generator=gen)
    centre, width, amp = u[:, :3] * n, 4 + 28 * u[:, 3], 2 * u[:, 4] - 1
    x = torch.arange(n, dtype=torch.float32, device="cuda")
    axis = [torch.exp(-0.5 * ((x[None] - centre[:, k:k + 1]) / width[:, None]) ** 2) for k in range(3)]
    re = torch.einsum("bz,by,bx->zyx", axis[0] * amp[:, None], axis[1], axis[2])
    noise = torch.empty((n, n, n, 2), dtype=torch.float32, device="cuda").uniform_(-1e-3, 1e-3, generator=gen)
    noise[..., 0] += re
    return torch.view_as_complex(noise)


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["kind"] == "uneven":
        sizes = _sizes(case)
        sig = _complex(gen, (sum(n ** 3 for n in sizes),))
        sigma = 1 + 7 * torch.rand(len(sizes), generator=gen, device="cuda").cpu()
        filt = torch.cat([_gaussian(n, float(s)).flatten() for n, s in zip(sizes, sigma)]).to(torch.complex64)
        return sig, filt
    n, b = case["n"], case["batch"]
    cube = (n, n, n)
    if case["kind"] == "transform":
        return None, _complex(gen, (b,) + cube)
    if case["kind"] == "host":
        return _complex(gen, (b,) + cube), _gaussian(n, 4.0 * n / 128).to(torch.complex64)
    sig = torch.cat([_blobs(gen, n)[None] for _ in range(b)]) if n == 512 else _complex(gen, (b,) + cube, normal=n == 256)
    if case["filter"] == "real":
        return sig, _gaussian(n, {512: 6.0, 128: 4.0}.get(n, n / 32))
    return sig, _complex(gen, ((b,) if case["filter"] == "pairs" else ()) + cube)


def _flags(case):
    return ((cg.NORMALIZE if case["normalize"] else 0) | (cg.TENSOR_SPLIT if case["split"] else 0)
            | {"shared": 0, "pairs": cg.FILTER_PER_SIGNAL, "real": cg.FILTER_REAL, "spectrum": cg.FILTER_IS_SPECTRUM}[case["filter"]])


def prepare(case, seed):
    sizes = sorted(set(_sizes(case))) if case["kind"] == "uneven" else [case["n"]]
    if set(sizes) - _tuned:
        cg.autotune([n for n in sizes if n not in _tuned], write_cache=False)
        _tuned.update(sizes)
    sig, filt = _inputs(case, seed)
    state = {"case": case}
    if case["kind"] == "uneven":
        offs = np.cumsum([0] + [n ** 3 for n in _sizes(case)])
        state["jobs"] = [(n, int(o), int(o), int(o)) for n, o in zip(_sizes(case), offs)]
    if case["kind"] == "transform":
        return {**state, "filt": filt, "out": torch.empty_like(filt)}
    if case["kind"] == "host":
        out = np.empty(tuple(sig.shape), np.complex64)
        out.fill(0)
        return {**state, "sig": sig.cpu().numpy(), "filt": filt.cpu().numpy(), "out": out}
    if case["kind"] == "conv" and case["filter"] == "spectrum":
        spec = torch.empty_like(filt)
        cg.filter_spectrum_device(case["n"], filt, spec, 1, torch.cuda.current_stream())
        filt = spec
    return {**state, "sig": sig, "filt": filt, "out": torch.empty_like(sig)}


def run(state):
    case, out = state["case"], state["out"]
    if case["kind"] == "host":
        if not cg.fpgaf_conv3D_svm_batch(case["n"], state["sig"], state["filt"], out, case["batch"]).valid:
            raise RuntimeError(cg.last_error())
        return out
    stream = torch.cuda.current_stream()
    if case["kind"] == "uneven":
        cg.conv3d_uneven_device(state["jobs"], state["sig"], state["filt"], out, cg.NORMALIZE, stream)
    elif case["kind"] == "transform":
        cg.filter_spectrum_device(case["n"], state["filt"], out, case["batch"], stream)
    else:
        cg.conv3d_device(case["n"], state["sig"], state["filt"], out, case["batch"], _flags(case), stream)
    return out


def work(case):
    """Inputs read and outputs written once; 5 N^3 log2(N^3) operations for each transform and 6 N^3 for each product."""
    if case["kind"] == "uneven":
        parts = [(n, 1, 1, 8) for n in _sizes(case)]
    else:
        n, b, kind = case["n"], case["batch"], case.get("filter")
        parts = [(n, b, b if kind == "pairs" else 1, 4 if kind == "real" else 8)]
    byts = flops = 0
    for n, b, nf, fbytes in parts:
        v, fft = n ** 3, 15 * n ** 3 * int(math.log2(n))
        if case["kind"] == "transform":
            byts += 16 * v * b
            flops += fft * b
            continue
        byts += 16 * v * b + fbytes * v * nf
        flops += (2 * fft + 6 * v) * b + (0 if case.get("filter") == "spectrum" else fft * nf)
    return {"bytes": byts, "flops": flops}


def exact(case, seed):
    sig, filt = _inputs(case, seed)

    def fft(x):
        return torch.fft.fftn(x.to(torch.complex128), dim=(-3, -2, -1))

    def conv(s, f, normalize):
        out = torch.empty(s.shape, dtype=torch.complex128, device=s.device)
        spec = fft(f) if f.dim() == 3 else None
        for i in range(s.shape[0]):
            out[i] = torch.fft.ifftn(fft(s[i]) * (fft(f[i]) if spec is None else spec), dim=(-3, -2, -1))
            if not normalize:
                out[i] *= s.shape[-1] ** 3
        return out

    if case["kind"] == "transform":
        return torch.stack([fft(f) for f in filt])
    if case["kind"] == "host":
        return conv(sig, filt, False).cpu().numpy()
    if case["kind"] == "uneven":
        out = torch.empty(sig.shape, dtype=torch.complex128, device="cuda")
        at = 0
        for n in _sizes(case):
            part = slice(at, at + n ** 3)
            out[part] = conv(sig[part].view(1, n, n, n), filt[part].view(n, n, n), True).flatten()
            at += n ** 3
        return out
    return conv(sig, filt, case["normalize"])
