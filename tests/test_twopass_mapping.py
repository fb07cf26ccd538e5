"""The two-pass transform's index maps, restated and checked on the CPU (twopass.cuh).

A cube of N^3 points goes through k_tp_fwd's tiles (radix-2 step of z, x, J points of y)
into tile order, through k_tp_mid's tiles (the rest of y and z, the product, back) and
through k_tp_inv's; here every tile is addressed by the kernels' own formulas and
transformed with numpy in complex128, so the result equals the FFT convolution only if
every map, step twiddle and slot is right. The exchange slots inside a tile are checked to
be a permutation of the tile.
"""
import numpy as np
import pytest

# N: (J rows of the outer tile, C interleaved columns of the middle tile)
SHAPES = {32: (8, 2), 64: (8, 4), 128: (16, 4), 256: (16, 2)}
SPLIT = {256: (16, 16), 128: (16, 8), 64: (8, 8), 32: (8, 4), 16: (4, 4)}


def _fwd(cube, j_rows, c_cols):
    """k_tp_fwd: natural order -> tile order, as (units, 2 lanes); every unit written once."""
    n = cube.shape[0]
    r, h = n // j_rows, n // 2
    w = np.exp(-2j * np.pi * np.arange(n) / n)
    out = np.full((n ** 3 // 2, 2), np.nan, complex)
    kx, j = np.arange(n)[:, None], np.arange(j_rows)[None, :]
    for y0 in range(r):
        for zz in range(h):
            p, q = cube[zz, y0::r], cube[zz + h, y0::r]  # rows y0 + R j
            lanes = np.stack([p + q, p - q], -1)
            t = np.fft.fft2(lanes, axes=(1, 0))          # [j'][kx][lane]
            t = t * np.stack([w[(y0 * j[0]) % n], w[(y0 * j[0] + zz) % n]], -1)[:, None, :]
            u = (((j // c_cols) * n + kx) * (r * h) + (y0 * h + zz)) * c_cols + j % c_cols
            assert np.isnan(out[u]).all()
            out[u] = t.transpose(1, 0, 2)
    assert not np.isnan(out).any()
    return out


def _mid(units, n, j_rows, c_cols, inverse=False):
    """Forward (or unnormalised inverse) transform of k_tp_mid's tiles [y0][zz][c] <-> [k2][kz'][c]."""
    t = units.reshape(-1, n // j_rows, n // 2, c_cols, 2)
    t = np.fft.ifft2(t, axes=(1, 2)) * (n // j_rows) * (n // 2) if inverse else np.fft.fft2(t, axes=(1, 2))
    return t.reshape(-1, 2)


def _inv(units, n, j_rows, c_cols):
    r, h = n // j_rows, n // 2
    w = np.exp(2j * np.pi * np.arange(n) / n)
    out = np.full((n, n, n), np.nan, complex)
    kx, j = np.arange(n)[:, None], np.arange(j_rows)[None, :]
    for y0 in range(r):
        for zz in range(h):
            u = (((j // c_cols) * n + kx) * (r * h) + (y0 * h + zz)) * c_cols + j % c_cols
            t = units[u].transpose(1, 0, 2)
            t = t * np.stack([w[(y0 * j[0]) % n], w[(y0 * j[0] + zz) % n]], -1)[:, None, :]
            t = np.fft.ifft2(t, axes=(1, 0)) * n * j_rows
            out[zz, y0::r], out[zz + h, y0::r] = t[..., 0] + t[..., 1], t[..., 0] - t[..., 1]
    assert not np.isnan(out).any()
    return out


@pytest.mark.parametrize("n", [32, 64])
def test_two_pass_convolution_restated(n):
    j_rows, c_cols = SHAPES[n]
    rng = np.random.default_rng(n)
    sig, filt = (rng.standard_normal((n, n, n)) + 1j * rng.standard_normal((n, n, n)) for _ in range(2))
    s = _mid(_fwd(sig, j_rows, c_cols), n, j_rows, c_cols)
    f = _mid(_fwd(filt, j_rows, c_cols), n, j_rows, c_cols)
    # a spectrum's place: tile (g, kx), unit (k2 H + kz') C + c holds kz = 2 kz' + lane, ky = g C + c + J k2
    spec = np.fft.fftn(sig)
    u = np.arange(n ** 3 // 2)
    tile, unit = u // (n // j_rows * (n // 2) * c_cols), u % (n // j_rows * (n // 2) * c_cols)
    k2, kzh, c = unit // (n // 2 * c_cols), unit // c_cols % (n // 2), unit % c_cols
    ky, kx = (tile // n) * c_cols + c + j_rows * k2, tile % n
    for lane in range(2):
        np.testing.assert_allclose(s[:, lane], spec[2 * kzh + lane, ky, kx], rtol=0, atol=1e-9 * n ** 1.5)
    got = _inv(_mid(s * f, n, j_rows, c_cols, inverse=True), n, j_rows, c_cols)
    ref = np.fft.ifftn(spec * np.fft.fftn(filt)) * n ** 3
    assert np.linalg.norm(got - ref) < 1e-12 * np.linalg.norm(ref)


def _tiles():
    for n, (j_rows, c_cols) in SHAPES.items():
        if n >= 128:
            yield n, j_rows, 1
            yield n // 2, n // j_rows, c_cols


@pytest.mark.parametrize("n,j_rows,c_cols", list(_tiles()))
def test_tile_slots(n, j_rows, c_cols):
    """The row exchange's slots (tilefft.cuh: ex_w by its writers, ex_r by its readers) and the
    column slots are permutations of the tile, both sides agree, and 8 consecutive lanes of
    each access hit 8 different 16-byte bank groups."""
    r1, r2 = SPLIT[n]
    t_row = n // 16
    nt = n * j_rows * c_cols // 16
    sw = min(r2, 8) - 1
    tid = np.arange(nt)
    c, t, row, colt = tid % c_cols, tid // c_cols % t_row, tid // (c_cols * t_row), tid // c_cols

    def unit(row, i, c):
        return (row * n + i) * c_cols + c

    def banks(u):
        for at in range(0, nt, 8):
            assert len(set(u[at:at + 8] % 8)) == 8
    written, read, cols = {}, {}, set()
    for i in range(16 // r1):
        for k1 in range(r1):
            u = unit(row, k1 * r2 + ((t + i * t_row) ^ (k1 & sw)), c)
            banks(u)
            written.update({int(a): (int(b), k1, int(d), int(e)) for a, b, d, e in zip(u, row, t + i * t_row, c)})
    for i in range(16 // r2):
        for tt in range(r2):
            k1 = t + i * t_row
            u = unit(row, k1 * r2 + (tt ^ (k1 & sw)), c)
            banks(u)
            read.update({int(a): (int(b), int(d), tt, int(e)) for a, b, d, e in zip(u, row, k1, c)})
    assert written == read and sorted(written) == list(range(n * j_rows * c_cols))
    for i in range(16 // j_rows):
        for j in range(j_rows):
            u = unit(j, colt + i * (nt // c_cols), c)
            banks(u)
            cols.update(u.tolist())
    assert cols == set(range(n * j_rows * c_cols))
