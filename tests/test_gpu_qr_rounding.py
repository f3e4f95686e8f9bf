"""The residual of the one-launch Householder QR: an entry takes one rounding an update.

Of k columns an entry goes through k / 2 updates on average while R is formed and k / 2
while Q is. Each rounds once at the size of the entry, an error of 0.41 of 2^-53 (root
mean square, for a spread of mantissas), independent of the others: |Q R - A| / |A| is
about 0.41 sqrt(k) 2^-53. Two roundings an update would make it 0.58 sqrt(k) 2^-53; the
bound lies half way."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k", [(512, 256), (256, 128), (1024, 256)])
@pytest.mark.parametrize("entry", ["ptn_zqr_keep", "ptn_zqr_keep_steps"])
def test_residual_of_one_rounding_an_update(m, k, entry):
    from pytreenet_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(m + k)
    square = 0.0
    for _ in range(4):
        A = rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k))
        a = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
        ro = torch.arange(m, dtype=torch.int64, device="cuda")
        R = torch.zeros(k * k, dtype=torch.complex128, device="cuda")
        w = torch.empty((lib.ptn_zqr_work_bytes(m, k) + 15) // 16, dtype=torch.complex128, device="cuda")
        assert getattr(lib, entry)(a.data_ptr(), ro.data_ptr(), m, k, m, R.data_ptr(), w.data_ptr(),
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        Q = a.cpu().numpy().T.astype(np.clongdouble)
        rest = Q @ R.cpu().numpy().reshape(k, k).astype(np.clongdouble) - A
        square += float((np.linalg.norm(rest.astype(complex)) / np.linalg.norm(A)) ** 2)
    assert (square / 4) ** 0.5 <= 0.5 * k ** 0.5 * 2.0 ** -53
