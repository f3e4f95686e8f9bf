"""Tensor-core contraction at the edges of its tiles and in every way its epilogue
stores: 64- and 128-column tiles, ragged rows and columns, several tiles per CTA, and
output layouts whose contiguous index is the column, the row, a pair of rows or a mix.

The products are formed from given BF16 planes. With small whole numbers in them every
FP32 sum is exact, and so must the complex128 output be; the plane output must be the
BF16 split of the complex128 one, entry for entry, whatever the layout and the numbers."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from pytreenet_gb300 import _lib
    return _lib.load()


def _modes(m, pairs):
    m.n = len(pairs)
    for i, (d, s) in enumerate(pairs):
        m.dim[i], m.stride_c[i] = d, s


def _offsets(pairs):
    o = np.zeros(1, dtype=np.int64)
    for d, s in pairs:
        o = (o[:, None] + np.arange(d, dtype=np.int64)[None, :] * s).reshape(-1)
    return o


def _layout(name, M, N):
    """(row modes, column modes, entries) of an output without overlaps."""
    r = lambda v, q: -(-v // q) * q
    if name == "rows":                   # columns contiguous
        return [(M, N)], [(N, 1)], M * N
    if name == "rows8":                  # the same, rows padded to 16 bytes
        return [(M, r(N, 8))], [(N, 1)], M * r(N, 8)
    if name == "columns":                # rows contiguous
        return [(M, 1)], [(N, M)], M * N
    if name == "pairs":                  # a leg of dimension 2 innermost, then the columns
        return [(M // 2, 2 * N), (2, 1)], [(N, 2)], M * N
    if name == "pairs8":
        return [(M // 2, r(2 * N, 8)), (2, 1)], [(N, 2)], (M // 2) * r(2 * N, 8)
    if name == "mixed":                  # rows of w d = 10
        return [(M // 2, 10), (2, 1)], [(N // 5, 5 * M), (5, 2)], M * N
    raise ValueError(name)


def _run(lib, A, B, M, N, K, L, kind, rows, cols, size):
    from pytreenet_gb300 import _lib
    d = _lib.CgemmDesc()
    ld = A.shape[-1]
    plane = -(-size // 8) * 8
    if kind == 0:
        C = torch.full((size,), 7.0, dtype=torch.complex128, device="cuda")
    else:
        C = torch.full((2 * L * plane,), 7.0, dtype=torch.bfloat16, device="cuda")
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    d.A, d.lda, d.a_plane, d.M, d.K = A.data_ptr(), ld, M * ld, M, K
    d.Bx, d.ldb, d.N, d.out_kind, d.levels = B.data_ptr(), ld, N, kind, L
    d.C, d.c_plane, d.status = C.data_ptr(), plane, st.data_ptr()
    _modes(d.m_out, rows)
    _modes(d.n_out, cols)
    assert lib.ptn_cgemm_bf16x3(ctypes.byref(d), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    assert int(st.item()) == 0
    idx = torch.from_numpy(_offsets(rows)[:, None] + _offsets(cols)[None, :]).cuda()
    if kind == 0:
        return C[idx]
    return C.view(2 * L, plane)[:, idx.reshape(-1)].view(2 * L, M, N)


@pytest.mark.parametrize("M,N,K", [(2, 8, 40), (130, 13, 65), (254, 65, 48), (258, 130, 100), (126, 66, 33),
                                   (1000, 90, 90), (640, 100, 320), (20000, 70, 48), (40000, 200, 40)])
@pytest.mark.parametrize("L", [2, 3])
@pytest.mark.parametrize("whole", [True, False])
def test_every_store_gives_the_same_entries(lib, M, N, K, L, whole):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    ld = -(-K // 8) * 8

    def draw(*shape):
        if whole:                        # |sums| <= 2 * 6 * 320 * 9 < 2^24
            return torch.randint(-3, 4, shape, device="cuda", generator=g).to(torch.bfloat16)
        return torch.randn(shape, device="cuda", generator=g).to(torch.bfloat16)
    A, B = draw(2 * L, M, ld), draw(3 * L, N, ld)
    B[0::3] = -B[2::3]
    want = None
    for name in ("rows", "rows8", "columns", "pairs", "pairs8", "mixed"):
        if name == "mixed" and N % 5:
            continue
        rows, cols, size = _layout(name, M, N)
        c = _run(lib, A, B, M, N, K, L, 0, rows, cols, size)
        if want is None:
            want = c
            if whole:
                a = (A[0::2].to(torch.complex128) + 1j * A[1::2].to(torch.complex128))[:, :, :K]
                b = (B[1::3].to(torch.complex128) + 1j * B[2::3].to(torch.complex128))[:, :, :K]
                assert torch.equal(c, sum(a[i] @ b[j].T for i in range(L) for j in range(L - i)))
        else:
            assert torch.equal(c, want), name
        p = _run(lib, A, B, M, N, K, L, 1, rows, cols, size)
        for part, x in ((0, want.real.float()), (1, want.imag.float())):
            for lv in range(L):
                piece = x.to(torch.bfloat16)
                assert torch.equal(p[2 * lv + part], piece), (name, lv)
                x = x - piece.float()


@pytest.mark.parametrize("K", [2, 4, 6, 10])
@pytest.mark.parametrize("N", [1, 50, 128])
@pytest.mark.parametrize("M,pad", [(2, 0), (254, 0), (600, 3), (600, 6), (40000, 0)])
@pytest.mark.parametrize("L", [2, 3])
def test_row_pairs_of_short_products(lib, K, N, M, pad, L):
    """Products with K <= 10 on the FP32 units: two rows an instruction and rows read in
    words must give what one row a thread gives (the complex128 output's kernel)."""
    g = torch.Generator(device="cuda").manual_seed(K + N)
    lda = K + pad
    rows, cols, size = _layout("pairs", M, N)
    plane = -(-M * lda // 8) * 8
    A = torch.randn((2 * L, plane), device="cuda", generator=g).to(torch.bfloat16)
    B = torch.randn((3 * L, N, -(-K // 8) * 8), device="cuda", generator=g).to(torch.bfloat16)
    B[0::3] = -B[2::3]
    got = {}
    for kind in (0, 1):
        from pytreenet_gb300 import _lib
        d = _lib.CgemmDesc()
        cp = -(-size // 8) * 8
        C = torch.zeros((size if kind == 0 else 2 * L * cp,), device="cuda",
                        dtype=torch.complex128 if kind == 0 else torch.bfloat16)
        st = torch.zeros(1, dtype=torch.int32, device="cuda")
        d.A, d.lda, d.a_plane, d.M, d.K = A.data_ptr(), lda, plane, M, K
        d.Bx, d.ldb, d.N, d.out_kind, d.levels = B.data_ptr(), B.shape[-1], N, kind, L
        d.C, d.c_plane, d.status = C.data_ptr(), cp, st.data_ptr()
        _modes(d.m_out, rows)
        _modes(d.n_out, cols)
        assert lib.ptn_cgemm_bf16x3(ctypes.byref(d), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        got[kind] = C if kind == 0 else C.view(2 * L, cp)[:, :size]
    for part, x in ((0, got[0].real.float()), (1, got[0].imag.float())):
        for lv in range(L):
            piece = x.to(torch.bfloat16)
            assert torch.equal(got[1][2 * lv + part], piece)
            x = x - piece.float()
