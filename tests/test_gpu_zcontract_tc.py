"""Complex128 contractions as digit products on the tensor cores (``ptn_zcontract_ws``)
against the FP64 kernels (``ptn_zcontract``) on the same operands.

Bound: an operand is rounded at 2^-55 of twice its row's largest entry after the
balancing along K (which moves entries by less than a factor 2 against each other),
2 K products per real output; the FP64 sum loses at most 2 K 2^-53 of the sum of
magnitudes. Together below K 2^-49 max|a| max|b| where B's rows are of one size."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(la, da, lb, db, lc, kl, a, b, c0=None, **kw):
    from pytreenet_gb300 import _lib
    from pytreenet_gb300.engine import Operand, Step, _stream_ptr
    lib = _lib.load()
    dims = {**dict(zip(la, da)), **dict(zip(lb, db))}
    shape = [dims[l] for l in lc]
    st = Step(Operand.contiguous(("fixed", None), la, da), Operand.contiguous(("fixed", None), lb, db), kl,
              Operand.contiguous(("fixed", None), lc, shape), **kw)
    c0 = torch.zeros(shape, dtype=torch.complex128, device="cuda") if c0 is None else c0
    d = st.desc
    d.A, d.B = a.data_ptr(), b.data_ptr()
    nbytes = int(lib.ptn_zcontract_work_bytes(ctypes.byref(d)))
    assert nbytes > 0, "the sizes must take the tensor-core path"
    work = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    plain, tc = c0.clone(), c0.clone()
    d.C = plain.data_ptr()
    assert lib.ptn_zcontract(ctypes.byref(d), _stream_ptr()) == 0
    d.C = tc.data_ptr()
    assert lib.ptn_zcontract_ws(ctypes.byref(d), work.data_ptr(), nbytes, _stream_ptr()) == 0
    torch.cuda.synchronize()
    return plain, tc


def _gauss(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, dtype=torch.complex128, device="cuda", generator=g)


# tiles of 128 x 32, stages of 16, chunks of 64, one split per 4096 K values,
# 1 GiB of digits per turn
@pytest.mark.parametrize("M,K,N", [(128, 64, 512), (129, 65, 400), (127, 63, 417), (4097, 17, 47), (65536, 10, 10),
                                   (33, 4113, 65), (90, 8100, 31), (640, 128, 128), (31, 200, 5000),
                                   (130000, 320, 8), (3000000, 2, 2)])
def test_zcontract_tc_sizes(M, K, N):
    a, b = _gauss((M, K), 1), _gauss((K, N), 2)
    plain, tc = _run(["m", "k"], [M, K], ["k", "n"], [K, N], ["m", "n"], ["k"], a, b)
    tol = K * 2.0 ** -49 * float(a.abs().max() * b.abs().max())
    assert float((plain - tc).abs().max()) <= tol


@pytest.mark.parametrize("kw", [{}, {"conj_a": True}, {"conj_b": True}, {"alpha": 0.5 - 2j, "beta": 1.0}])
@pytest.mark.parametrize("lc", [["d", "a", "c", "b"], ["a", "b", "c", "d"]])
def test_zcontract_tc_modes(kw, lc):
    dims = {"a": 13, "k": 7, "b": 22, "l": 19, "c": 11, "d": 30}
    la, lb = ["a", "k", "b", "l"], ["l", "c", "k", "d"]
    a, b = _gauss([dims[l] for l in la], 3), _gauss([dims[l] for l in lb], 4)
    c0 = _gauss([dims[l] for l in lc], 5)
    plain, tc = _run(la, [dims[l] for l in la], lb, [dims[l] for l in lb], lc, ["k", "l"], a, b, c0, **kw)
    tol = 133 * 2.0 ** -49 * float(a.abs().max() * b.abs().max()) * abs(kw.get("alpha", 1.0)) + 2.0 ** -50
    assert float((plain - tc).abs().max()) <= tol


def test_zcontract_tc_range_of_magnitudes():
    """Operands graded against each other along K, rows and columns of any size,
    rows of zeros, denormals, and entries that are not finite."""
    M, K, N = 256, 96, 160
    a, b = _gauss((M, K), 6), _gauss((K, N), 7)
    grade = torch.exp(-0.6 * torch.arange(K, dtype=torch.float64, device="cuda"))
    rows = torch.exp(40 * torch.randn(M, 1, dtype=torch.float64, device="cuda",
                                      generator=torch.Generator(device="cuda").manual_seed(8)))
    args = (["m", "k"], [M, K], ["k", "n"], [K, N], ["m", "n"], ["k"])
    tol = K * 2.0 ** -49 * float(a.abs().max() * b.abs().max())
    plain, tc = _run(*args, a * grade, b / grade[:, None])
    assert float((plain - tc).abs().max()) <= tol
    plain, tc = _run(*args, a * rows, b)
    assert float(((plain - tc).abs() / rows).max()) <= tol
    a[5] = 0
    a[6] *= 1e-310
    a[7] *= 1e-200
    plain, tc = _run(*args, a, b)
    assert torch.equal(tc[5], torch.zeros_like(tc[5]))
    assert torch.equal(tc[6], plain[6])                 # summed in FP64
    assert float((plain - tc)[7].abs().max()) <= tol * 1e-200
    a[3, 4], a[9, 2], b[8, 11] = complex("nan"), complex("inf"), complex("-inf")
    plain, tc = _run(*args, a, b)
    p, t = torch.view_as_real(plain), torch.view_as_real(tc)
    assert torch.equal(torch.isnan(p), torch.isnan(t)) and torch.equal(torch.isinf(p), torch.isinf(t))
    assert not torch.isfinite(p[9]).any() and torch.isfinite(p[0, 0]).all()


def test_zcontract_tc_repeats_and_scratch():
    """The same bits on every run, and the FP64 kernels when the scratch is short."""
    from pytreenet_gb300 import _lib
    from pytreenet_gb300.engine import Operand, Step, _stream_ptr
    lib = _lib.load()
    a, b = _gauss((300, 2000), 9), _gauss((2000, 70), 10)
    st = Step(Operand.contiguous(("fixed", None), ["m", "k"], [300, 2000]),
              Operand.contiguous(("fixed", None), ["k", "n"], [2000, 70]), ["k"],
              Operand.contiguous(("fixed", None), ["m", "n"], [300, 70]))
    d = st.desc
    nbytes = int(lib.ptn_zcontract_work_bytes(ctypes.byref(d)))
    work = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    out = [torch.empty(300, 70, dtype=torch.complex128, device="cuda") for _ in range(4)]
    d.A, d.B = a.data_ptr(), b.data_ptr()
    for c, n in zip(out, (nbytes, nbytes, nbytes - 1, 0)):
        d.C = c.data_ptr()
        assert lib.ptn_zcontract_ws(ctypes.byref(d), work.data_ptr() if n else None, n, _stream_ptr()) == 0
    torch.cuda.synchronize()
    assert torch.equal(out[0], out[1])
    ref = a.cpu().numpy() @ b.cpu().numpy()
    for c in out:
        assert np.abs(c.cpu().numpy() - ref).max() < 1e-11
