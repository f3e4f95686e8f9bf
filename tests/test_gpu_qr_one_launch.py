"""One-launch Householder QR at the edges of its row split and of the number range.

The kernel gives a thread 1, 2, 4, 8 or 16 rows, and a CTA an even or odd number of
columns. Checked against the properties that define the factorisation (oracle:
LAPACK's conventions, util/tensor_splitting.py:60-107): Q R = A, Q^H Q = 1, R upper
triangular with a real diagonal of the sign -sign(Re a_jj) in column 0.
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


@pytest.fixture(scope="module")
def lib():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from pytreenet_gb300 import _lib
    return _lib.load()


def _qr(lib, A):
    m, k = A.shape
    a = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    ro = torch.arange(m, dtype=torch.int64, device="cuda")
    R = torch.full((k * k,), 7.0, dtype=torch.complex128, device="cuda")
    w = torch.empty((lib.ptn_zqr_work_bytes(m, k) + 15) // 16, dtype=torch.complex128, device="cuda")
    st = lib.ptn_zqr_keep(a.data_ptr(), ro.data_ptr(), m, k, m, R.data_ptr(), w.data_ptr(),
                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    return a.cpu().numpy().T, R.cpu().numpy().reshape(k, k)


@pytest.mark.parametrize("m,k", [(1, 1), (1, 3), (3, 5), (127, 3), (128, 64), (129, 2), (255, 31), (257, 256),
                                 (513, 7), (1025, 3), (2047, 5), (2048, 160)])
@pytest.mark.parametrize("scale", [1.0, 1e-130, 1e-148, 1e147])
def test_one_launch_qr_factorises(lib, m, k, scale):
    """Backward error of Householder QR is at most a small multiple of m k eps; the
    rounding of the sums is random, so sqrt(m) k eps with a factor of 16 is safe. The
    two small scales and the large one square to near the ends of the number range:
    at 1e-148 to 1e-296, so entries a factor 1e7 below lose digits to gradual underflow,
    none here."""
    rng = np.random.default_rng(m * 1000 + k)
    A = scale * (rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k)))
    Q, R = _qr(lib, A)
    p = min(m, k)
    tol = 16 * np.sqrt(m) * k * EPS
    assert np.abs(Q[:, :p].conj().T @ Q[:, :p] - np.eye(p)).max() <= tol
    assert np.linalg.norm((Q[:, :p] @ R[:p] - A) / scale) <= tol * np.linalg.norm(A / scale)
    assert not np.any(np.tril(R, -1)) and not np.any(R[p:]) and not np.any(Q[:, p:])
    d = np.diag(R)[: p - 1 if p == m else p]
    assert not np.any(d.imag)
    assert len(d) == 0 or np.sign(d[0].real) == -np.sign(A[0, 0].real)


def test_one_launch_qr_of_zero_columns_and_nan(lib):
    """A zero column leaves tau = 0 (Q column = unit vector, R entry exactly 0); NaN
    inputs with any payload come back as NaN and end the call."""
    A = np.zeros((40, 6), dtype=complex)
    A[:, 0] = 1.0
    Q, R = _qr(lib, A)
    assert not np.any(R[1:]) and np.isfinite(Q).all()
    assert np.abs(Q.conj().T @ Q - np.eye(6)).max() <= 16 * np.sqrt(40) * 6 * EPS
    B = np.random.default_rng(0).standard_normal((40, 6)).astype(complex)
    B.view(np.uint64).reshape(40, 6, 2)[5, 2, :] = np.uint64(0xFFFFFFFFFFFFFFFF)
    Q, R = _qr(lib, B)
    assert np.isnan(R[2, 2]) and np.isfinite(R[:2, :2]).all()
