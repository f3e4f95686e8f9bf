"""Conversion of complex128 operands into BF16 pieces: the integer rounding of the leading
piece at its edges (ties, carries into the exponent, zeros, both ends of its range), and
every way the kernels index and store (tiles, two and four entries a thread, odd leading
dimensions)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from pytreenet_gb300 import _lib
    return _lib.load()


def _round8(x):
    """To eight significant bits, ties to even (exact in FP64)."""
    m, e = np.frexp(x)
    return np.ldexp(np.rint(m * 256.0), e - 8)


def _pieces(x, L):
    out = [_round8(x)]
    r = (x - out[0]).astype(np.float32)          # exact in FP64, rounded once
    for _ in range(1, L):
        b = _round8(r.astype(np.float64))
        out.append(b)
        r = (r - b.astype(np.float32)).astype(np.float32)
    return out


def _values(rng, n):
    x = rng.standard_normal(n)
    q = rng.integers(0, 8, n)
    k = rng.integers(-62, 100, n)
    x[q == 0] = np.where(rng.random(np.sum(q == 0)) < 0.5, 0.0, -0.0)
    m = q == 1                                    # at and beside ties
    x[m] = np.ldexp(1 + (2 * rng.integers(0, 128, m.sum()) + 1) / 256.0
                    + rng.integers(-1, 2, m.sum()) * 2.0 ** -52, k[m])
    m = q == 2                                    # just below and at a power of two
    x[m] = np.ldexp(1 - rng.integers(0, 3, m.sum()) * 2.0 ** -53, k[m])
    m = q == 3                                    # few or no bits below the eighth
    x[m] = -np.ldexp(1 + rng.integers(0, 128, m.sum()) / 128.0 + rng.integers(0, 2, m.sum()) * 2.0 ** -50, k[m])
    m = q == 4
    x[m] = np.ldexp(x[m], k[m])
    return x


@pytest.mark.parametrize("rows,cols,pad", [
    ([(7, 13)], [(13, 1)], 0), ([(64, 52)], [(52, 1)], 4), ([(50, 54)], [(54, 1)], 1), ([(33, 66)], [(66, 1)], 2),
    ([(600, 1)], [(130, 600)], 6), ([(601, 1)], [(131, 601)], 0), ([(300, 2), (2, 1)], [(100, 600)], 4),
    ([(3, 1), (5, 60)], [(4, 15), (5, 3)], 4), ([(40, 1)], [(40, 40)], 0), ([(1, 1)], [(1, 1)], 7)])
@pytest.mark.parametrize("L", [2, 3])
@pytest.mark.parametrize("conj", [0, 1])
def test_pieces_are_the_rounded_ones(lib, rows, cols, pad, L, conj):
    from pytreenet_gb300 import _lib
    R, K = (int(np.prod([d for d, _ in m])) for m in (rows, cols))
    off = [np.zeros(1, dtype=np.int64), np.zeros(1, dtype=np.int64)]
    for i, m in enumerate((rows, cols)):
        for d, s in m:
            off[i] = (off[i][:, None] + np.arange(d)[None, :] * s).reshape(-1)
    idx = off[0][:, None] + off[1][None, :]
    rng = np.random.default_rng(R + K)
    src = np.empty(idx.max() + 1, dtype=complex)
    src.real, src.imag = _values(rng, src.size), _values(rng, src.size)
    dev = torch.from_numpy(src).cuda()
    x = src[idx]
    want = [_pieces(x.real, L), _pieces(-x.imag if conj else x.imag, L)]
    ld = K + pad
    plane = -(-R * ld // 8) * 8
    for expand in (False, True):
        n = 3 * L * R * ld if expand else 2 * L * plane
        dst = torch.full((n,), 7.0, dtype=torch.bfloat16, device="cuda")
        d = _lib.ConvertDesc()
        d.src, d.dst, d.ld, d.plane, d.conj, d.levels = dev.data_ptr(), dst.data_ptr(), ld, plane, conj, L
        for md, m in ((d.rows, rows), (d.cols, cols)):
            md.n = len(m)
            for i, (a, b) in enumerate(m):
                md.dim[i], md.stride_a[i] = a, b
        fn = lib.ptn_expand_b if expand else lib.ptn_to_planes
        assert fn(ctypes.byref(d), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        got = dst.double().cpu().numpy()
        for lv in range(L):
            if expand:
                blocks = got.reshape(L, 3, R, ld)[lv, :, :, :]
                pairs = [(blocks[0], -want[1][lv]), (blocks[1], want[0][lv]), (blocks[2], want[1][lv])]
            else:
                planes = [got[(2 * lv + c) * plane:][:R * ld].reshape(R, ld) for c in (0, 1)]
                pairs = [(planes[0], want[0][lv]), (planes[1], want[1][lv])]
            for have, ref in pairs:
                assert np.array_equal(have[:, :K], ref)
                assert np.all(have[:, K:] == 7.0)          # the padding is left alone
