"""The FP64 contraction kernel for few outputs (K slices in a CTA, clusters over K)
where its launch shape changes, against torch. Each side adds K complex products:
at most 4 K 2^-53 of the sum of magnitudes, K max|a| max|b| sqrt(2)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (1, 1, 7), (3, 2, 8), (2, 2, 255), (2, 2, 256), (1, 1, 4095), (2, 2, 4097),
                                   (13, 13, 1014), (16, 16, 64), (257, 1, 511), (33, 31, 127), (64, 64, 2500),
                                   (65, 64, 2500), (128, 129, 16), (300, 700, 3), (1, 5000, 33), (2, 3, 70001)])
@pytest.mark.parametrize("conj,beta", [(False, 0.0), (True, 1.0)])
def test_zcontract_few_outputs(M, N, K, conj, beta):
    from pytreenet_gb300 import _lib
    from pytreenet_gb300.engine import Operand, Step, _stream_ptr
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(M + 7 * N + 13 * K)
    # K in two modes where it factors, the output transposed
    k2 = next((d for d in (3, 2) if K % d == 0 and K > d), 1)
    a = torch.randn(K // k2, M, k2, dtype=torch.complex128, device="cuda", generator=g)
    b = torch.randn(k2, N, K // k2, dtype=torch.complex128, device="cuda", generator=g)
    c0 = torch.randn(N, M, dtype=torch.complex128, device="cuda", generator=g)
    st = Step(Operand.contiguous(("fixed", None), ["k", "m", "l"], [K // k2, M, k2]),
              Operand.contiguous(("fixed", None), ["l", "n", "k"], [k2, N, K // k2]), ["k", "l"],
              Operand.contiguous(("fixed", None), ["n", "m"], [N, M]), conj_b=conj, beta=beta)
    st.desc.A, st.desc.B = a.data_ptr(), b.data_ptr()
    out = []
    for _ in range(2):
        c = c0.clone()
        st.desc.C = c.data_ptr()
        assert lib.ptn_zcontract(ctypes.byref(st.desc), _stream_ptr()) == 0
        out.append(c)
    ref = torch.einsum("kml,lnk->nm", a, b.conj() if conj else b) + beta * c0
    tol = 2 * 4 * (K + 2) * 2.0 ** -53 * (K * 2.0 ** 0.5 * float(a.abs().max() * b.abs().max())
                                          + beta * float(c0.abs().max()))
    assert float((out[0] - ref).abs().max()) <= tol
    if M * N <= 4096:
        assert torch.equal(out[0], out[1])
