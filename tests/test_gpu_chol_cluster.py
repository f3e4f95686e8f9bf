"""The k x k factors of CholeskyQR2 at the edges of their blocks: one block and one
CTA up to k = 32, then a cluster of eight with 3 to 36 blocks, the last one padded."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
EPS32 = np.finfo(np.float32).eps


@pytest.fixture(scope="module")
def lib():
    from pytreenet_gb300 import _lib
    return _lib.load()


def _chol(lib, G, ldg, ratio=1e-3, series=0, tol=0.0):
    from pytreenet_gb300.engine import _stream_ptr
    k = G.shape[0]
    pad = np.full((k, ldg), np.nan + 0j)
    pad[:, :k] = G
    Gd = torch.from_numpy(pad).cuda()
    R = torch.full((k, k), 5.0, dtype=torch.complex128, device="cuda")
    Ri = torch.full_like(R, 5.0)
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    work = torch.zeros((int(lib.ptn_zchol_work_bytes(k)) + 15) // 16, dtype=torch.complex128, device="cuda")
    assert lib.ptn_zchol_upper(Gd.data_ptr(), ldg, k, R.data_ptr(), Ri.data_ptr(), ratio, series, tol,
                               st.data_ptr(), work.data_ptr(), _stream_ptr()) == 0
    return R.cpu().numpy(), Ri.cpu().numpy(), int(st.item())


@pytest.mark.parametrize("k", [1, 2, 31, 32, 33, 64, 65, 97, 255, 256])
def test_cluster_cholesky(lib, k):
    """Cholesky in FP32: |R^H R - G| <= c k eps |G|, c of order one (4 k terms a product,
    errors of random sign: 4 sqrt(k) + 8 covers it); |R R^-1 - 1| that times cond(R)."""
    rng = np.random.default_rng(k)
    A = (rng.standard_normal((2 * k + 1, k)) + 1j * rng.standard_normal((2 * k + 1, k))) / np.sqrt(2 * k)
    G = A.conj().T @ A
    R, Ri, st = _chol(lib, G, k + 3)
    assert st == 0
    assert not np.any(np.tril(R, -1)) and not np.any(np.tril(Ri, -1))
    tol = (4 * np.sqrt(k) + 8) * EPS32
    assert np.linalg.norm(R.conj().T @ R - G) <= tol * np.linalg.norm(G)
    assert np.linalg.norm(R @ Ri - np.eye(k)) <= tol * np.sqrt(k) * np.linalg.cond(R)
    # a pivot that is not positive, in the last column and in the first, and a small one
    for c in (0, k - 1):
        B = G.copy()
        B[c, c] = -1.0
        assert _chol(lib, B, k)[2] == 5
        B[c, c] = np.nan
        assert _chol(lib, B, k)[2] == 5
    if k > 1:
        assert _chol(lib, G, k, ratio=0.999)[2] == 5


@pytest.mark.parametrize("k", [1, 32, 33, 200, 256])
def test_first_order_factor(lib, k):
    """R = 1 + U, R^-1 = 1 - U from the Hermitian part, to FP64 rounding."""
    rng = np.random.default_rng(k)
    E = 1e-6 * (rng.standard_normal((k, k)) + 1j * rng.standard_normal((k, k)))
    H = 0.5 * (E + E.conj().T)
    R, Ri, st = _chol(lib, np.eye(k) + E, k + 1, series=1, tol=1e-3)
    U = np.triu(H, 1) + 0.5 * np.diag(np.diag(H).real)
    assert st == 0
    assert np.abs(R - np.eye(k) - U).max() <= 4e-16 and np.abs(Ri - np.eye(k) + U).max() <= 4e-16


@pytest.mark.parametrize("k", [1, 31, 32, 33, 130, 257])
def test_triangular_products(lib, k):
    """Sums of at most k products in FP64; entries below the diagonal are not read."""
    from pytreenet_gb300.engine import _stream_ptr
    rng = np.random.default_rng(k)
    A, B = (np.triu(rng.standard_normal((k, k)) + 1j * rng.standard_normal((k, k))) for _ in range(2))
    low = np.tril(np.full((k, k), np.nan + 0j), -1)
    Ad, Bd = torch.from_numpy(A + low).cuda(), torch.from_numpy(B + low).cuda()
    C, W = torch.full_like(Ad, 3.0), torch.full_like(Ad, 3.0)
    tol = 8 * np.finfo(float).eps * (np.abs(A) @ np.abs(B) + 1) * np.sqrt(k)
    assert lib.ptn_ztri_mul_upper(Ad.data_ptr(), Bd.data_ptr(), C.data_ptr(), k, _stream_ptr()) == 0
    got = C.cpu().numpy()
    assert np.all(np.abs(got - A @ B) <= tol) and not np.any(np.tril(got, -1))
    # R = B (2 - A B)
    assert lib.ptn_ztri_inv_newton(Ad.data_ptr(), Bd.data_ptr(), C.data_ptr(), W.data_ptr(), k, _stream_ptr()) == 0
    got = C.cpu().numpy()
    bound = 2 * np.abs(B) + np.abs(B) @ (np.abs(A) @ np.abs(B)) + 1
    assert np.all(np.abs(got - (2 * B - B @ (A @ B))) <= 16 * np.finfo(float).eps * np.sqrt(k) * bound)
