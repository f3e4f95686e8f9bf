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


@pytest.mark.parametrize("M,N,K,digits", [(1, 1, 1 << 22, False), (2, 3, 1 << 20, False), (16, 16, 65536, False),
                                          (1, 256, 20000, False), (257, 1, 20000, True), (64, 64, 4096, True),
                                          (128, 32, 1 << 24, False)])
def test_padding_and_workspace_keep_the_fp64_kernels(M, N, K, digits):
    """Where padding to a tile or the workspace would cost more than the FP64 kernels, no
    workspace is asked for, and the call with one still gives the product."""
    from pytreenet_gb300 import _lib
    from pytreenet_gb300.engine import Operand, Step
    lib = _lib.load()
    s = Step(Operand.contiguous(("fixed", None), ["m", "k"], [M, K]),
             Operand.contiguous(("fixed", None), ["n", "k"], [N, K]), ["k"],
             Operand.contiguous(("fixed", None), ["m", "n"], [M, N]))
    d = s.desc
    assert (int(lib.ptn_zcontract_work_bytes(ctypes.byref(d))) > 0) == digits
    if M * K > 1 << 25:
        return
    g = torch.Generator(device="cuda").manual_seed(K)
    A = torch.randn((M, K), dtype=torch.complex128, device="cuda", generator=g)
    B = torch.randn((N, K), dtype=torch.complex128, device="cuda", generator=g)
    C = torch.zeros((M, N), dtype=torch.complex128, device="cuda")
    ws = torch.empty(1 << 26, dtype=torch.uint8, device="cuda")
    d.A, d.B, d.C = A.data_ptr(), B.data_ptr(), C.data_ptr()
    assert lib.ptn_zcontract_ws(ctypes.byref(d), ws.data_ptr(), ws.numel(),
                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    ref = A @ B.T
    # sums of K terms of random sign in FP64, in whatever order
    scale = A.norm(dim=1)[:, None] * B.norm(dim=1)[None, :]
    assert ((C - ref).abs() <= 2.0 ** -50 * K ** 0.5 * scale).all()
