"""Complex128 contractions on the tensor cores with K around the length of one K split of
the operand conversion, where its offset table is largest, and far past it."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(2432, 256, 3968), (2432, 256, 3969), (2432, 256, 4033), (2432, 256, 4096),
                                   (2432, 256, 4097), (2432, 256, 7937), (1280, 256, 65536)])
def test_long_k(M, N, K):
    """Both sums round at 2^-53 of their terms' size; 2-norms of products of Gaussian
    operands differ by less than sqrt(K) 2^-53 relative, 1e-13 here."""
    from pytreenet_gb300 import _lib
    from pytreenet_gb300.engine import Operand, Step
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(K)
    A = torch.randn((M, K), dtype=torch.complex128, device="cuda", generator=g)
    B = torch.randn((N, K), dtype=torch.complex128, device="cuda", generator=g)
    C = torch.zeros((M, N), dtype=torch.complex128, device="cuda")
    s = Step(Operand.contiguous(("fixed", A), ["m", "k"], [M, K]), Operand.contiguous(("fixed", B), ["n", "k"], [N, K]),
             ["k"], Operand.contiguous(("fixed", C), ["m", "n"], [M, N]))
    d = s.desc
    d.A, d.B, d.C = A.data_ptr(), B.data_ptr(), C.data_ptr()
    nb = int(lib.ptn_zcontract_work_bytes(ctypes.byref(d)))
    assert nb > 0
    ws = torch.empty(nb + 256, dtype=torch.uint8, device="cuda")
    assert lib.ptn_zcontract_ws(ctypes.byref(d), ws.data_ptr(), nb,
                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    ref = A @ B.T
    assert (C - ref).norm().item() <= 1e-13 * ref.norm().item()
