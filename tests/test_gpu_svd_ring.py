"""The Jacobi SVD as a ring of CTAs (8 columns and more, up to 512 rows): edges of
its sizes against NumPy. Bounds: the iteration stops when every pair is
orthogonal to 8 sqrt(m) 2^-53, so U and V are orthonormal to n times that, and the
singular values and U S V^H follow to the same multiple of the largest one;
each column has gone through ~10 n rotations of 2^-52 rounding each."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _svd(A):
    from pytreenet_gb300 import _lib
    from pytreenet_gb300.engine import _stream_ptr
    lib = _lib.load()
    m, n = A.shape
    a = torch.from_numpy(np.ascontiguousarray(A, dtype=np.complex128)).cuda()
    U = torch.full((n * m,), float("nan"), dtype=torch.complex128, device="cuda")
    V = torch.full((n * n,), float("nan"), dtype=torch.complex128, device="cuda")
    S = torch.zeros(n + 1, dtype=torch.float64, device="cuda")
    # scratch that a previous call may have left anything in
    w = torch.full(((int(lib.ptn_zsvd_work_bytes(m, n)) + 15) // 16,), complex(1.0, 3.0), dtype=torch.complex128,
                   device="cuda")
    d = _lib.SvdDesc(a.data_ptr(), m, n, n, 1, U.data_ptr(), m, S.data_ptr(), V.data_ptr(), n, w.data_ptr(),
                     S[n:].data_ptr())
    out = []
    for _ in range(2):                                  # the second call finds the first one's scratch
        assert lib.ptn_zsvd_jacobi(ctypes.byref(d), _stream_ptr()) == 0
        h = S.cpu()
        assert int(h[n:].view(torch.int32)[0]) == 0
        out.append((U.cpu().numpy().reshape(n, m).T, h[:n].numpy().copy(), V.cpu().numpy().reshape(n, n).T))
    for x, y in zip(*out):
        assert np.array_equal(x, y, equal_nan=True)
    return out[0]


@pytest.mark.parametrize("m,n", [(8, 8), (9, 9), (127, 10), (128, 127), (129, 128), (257, 33), (512, 64), (130, 130),
                                 (310, 307), (8, 7), (513, 12)])
def test_svd_ring_sizes(m, n):
    rng = np.random.default_rng(m * 1000 + n)
    A = rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    U, S, V = _svd(A)
    eps = 8 * np.sqrt(m) * 2.0 ** -53 * n + 10 * n * 2.0 ** -52
    assert np.abs(U.conj().T @ U - np.eye(n)).max() < eps
    assert np.abs(V.conj().T @ V - np.eye(n)).max() < eps
    assert np.abs((U * S) @ V.conj().T - A).max() < eps * S[0]
    assert np.abs(S - np.linalg.svd(A, compute_uv=False)).max() < eps * S[0]


def test_svd_ring_rank_scale_and_zeros():
    rng = np.random.default_rng(5)
    n = 40
    G = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    low = (rng.standard_normal((n, 3)) + 0j) @ rng.standard_normal((3, n))
    graded = G * np.exp(-0.7 * np.arange(n))
    eps = 8 * np.sqrt(n) * 2.0 ** -53 * n + 10 * n * 2.0 ** -52
    for A in (low, graded, G * 1e-170, G * 1e200, np.zeros((n, n)), np.diag(np.arange(1.0, n + 1))):
        U, S, V = _svd(A)
        top = max(np.abs(A).max() * n, 1e-300)
        assert np.abs(V.conj().T @ V - np.eye(n)).max() < eps
        assert np.abs(((U * (S / top)) @ V.conj().T) - A / top).max() < eps
        assert np.all(np.diff(S) <= 0)
    G[3, 4] = np.nan                                    # ends, and says so in the singular values
    assert not np.isfinite(_svd(G)[1]).all()
