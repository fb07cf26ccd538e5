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
SHAPES = {32: (16, 16), 64: (16, 8), 128: (16, 4), 256: (16, 2)}


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


def _banks(units):
    for at in range(0, len(units), 8):
        assert len(set(units[at:at + 8] % 8)) == 8


@pytest.mark.parametrize("n,pad", [(32, 2), (64, 4), (128, 4), (256, 0)])
def test_outer_tile_slots(n, pad):
    """The outer tile's row exchange (written by ex_w, read by ex_r) and its column slots are
    permutations of the tile, both sides agree, and 8 consecutive lanes of each access hit 8
    different 16-byte bank groups."""
    j_rows, r2 = SHAPES[n][0], n // 16
    nt, sw = n * j_rows // 16, min(r2, 8) - 1
    tid = np.arange(nt)
    t, row = tid % r2, tid // r2
    written, read, cols = {}, {}, set()
    for k1 in range(16):
        u = row * (n + pad) + k1 * r2 + (t ^ (k1 & sw))
        _banks(u)
        written.update({int(a): (int(b), k1, int(c)) for a, b, c in zip(u, row, t)})
    for i in range(16 // r2):
        for tt in range(r2):
            k1 = t + i * r2
            u = row * (n + pad) + k1 * r2 + (tt ^ (k1 & sw))
            _banks(u)
            read.update({int(a): (int(b), int(c), tt) for a, b, c in zip(u, row, k1)})
    rows = {j * (n + pad) + x for j in range(j_rows) for x in range(n)}
    assert written == read and set(written) == rows
    for i in range(16 // j_rows):
        for j in range(j_rows):
            u = j * (n + pad) + tid + i * nt
            _banks(u)
            cols.update(u.tolist())
    assert cols == rows


def _trip(regs, col_of, reg_of):
    """rows-shape store, fragment-shape load of one warp's 32 lanes x 64 columns. regs: {(lane,
    label): value}; col_of(label): its column; returns {(lane, register): value}."""
    cell = {(lane, col_of(label)): v for (lane, label), v in regs.items()}
    out = {}
    for lane in range(32):
        for half in range(2):
            for rep in range(8):
                for q in range(4):
                    row, col = 16 * half + lane // 4 + 8 * (q >> 1), 8 * rep + 2 * (lane % 4) + (q & 1)
                    out[(lane, half * 32 + rep * 4 + q)] = cell[(row, col)]
    return out


@pytest.mark.parametrize("n", [64, 128, 256])
def test_middle_tile_exchange(n):
    """Two trips through TMEM take unit (k1) of lane (l4..l0) to lane (l0, k1), register
    s = (l4 l3 l2 l1); the twiddles between them are those of (t, k1); the shared-memory slots
    that follow are a permutation of the warp's rows and free of bank conflicts."""
    c_cols, r2 = SHAPES[n][1], n // 32
    col1 = lambda k, w: (k >> 2) << 1 | (k >> 1 & 1) << 3 | w << 4 | (k & 1) << 5
    frag1 = lambda m, w: (m >> 3) << 5 | (m & 1) << 4 | w << 3 | (m >> 1 & 1) << 2 | (m >> 2 & 1) << 1
    col2 = lambda m, w: (m >> 3) << 5 | (m >> 2 & 1) << 4 | w << 3 | (m & 3) << 1
    frag2 = lambda s, w: (s >> 1 & 1) << 5 | (s >> 2) << 3 | w << 2 | (s & 1) << 1
    first = {(lane, (k, w, h)): (lane, k, w, h) for lane in range(32) for k in range(16) for w in range(2) for h in range(2)}
    a = _trip(first, lambda x: col1(x[0], x[1]) + x[2], None)
    between = {}
    for lane in range(32):
        for m in range(16):
            for w in range(2):
                for h in range(2):
                    from_lane, k, w2, h2 = a[(lane, frag1(m, w) + h)]
                    q = (lane >> 3) * 4 + (lane & 3)  # the table's entry m 16 + q is for this t and k1
                    s = (m >> 2) << 2 | q >> 2
                    assert (from_lane >> 1, k, w2, h2) == (s, (q & 3) << 2 | (m & 3), w, h)
                    between[(lane, (m, w, h))] = (from_lane, k, w, h)
    b = _trip(between, lambda x: col2(x[0], x[1]) + x[2], None)
    for lane in range(32):
        for s in range(16):
            for w in range(2):
                for h in range(2):
                    assert b[(lane, frag2(s, w) + h)] == (s << 1 | lane >> 4, lane & 15, w, h)
    # lane before = (row, t, c) = 16 row + C t + c; butterfly i's input t is unit_of(i, t)
    hc = c_cols // 2
    unit_of = lambda i, t: (i // hc) * 8 + t * hc + i % hc
    slots = set()
    for i in range(16 // r2):
        for k2 in range(r2):
            u = []
            for lane in range(32):
                l0 = lane >> 4
                row, c = i // hc, (i % hc) * 2 + l0
                for t in range(r2):
                    assert unit_of(i, t) << 1 | l0 == 16 * row + c_cols * t + c
                kx = (lane & 15) + 16 * k2
                u.append(row * (n // 2) * c_cols + kx * c_cols + (c ^ ((kx * c_cols // 8) & (c_cols - 1))))
            _banks(np.array(u))
            slots.update(u)
    assert slots == set(range(n * c_cols))
