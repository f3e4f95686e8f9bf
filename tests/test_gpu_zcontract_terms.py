"""Complex128 contractions on the tensor cores hold every output to its own terms, as
the FP64 kernels do: operands whose rows and columns span many powers of two, with
zeros where the other operand is large.

Bound, with S = sum_k |a_mk| |b_kn| of an output: the FP64 sum of 2 K products per part
loses at most (2 K + 2) 2^-53 S in a part, below K 2^-51 S in the modulus. Digits are kept
where S is at least 2^-9 of the product of the row's and the column's power of two;
rounding both operands at 2^-64 of it and leaving out the digit products below loses
at most 18 K 2^-64 of it in a part, below K 2^-50 S in the modulus. Together K 2^-49 S."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _contract(a, b, tc, transposed=False, alpha=1.0, beta=0.0, c0=None):
    from pytreenet_gb300 import _lib
    from pytreenet_gb300.engine import Operand, Step, _stream_ptr
    lib = _lib.load()
    (M, K), N = a.shape, b.shape[1]
    lc, shape = (["n", "m"], [N, M]) if transposed else (["m", "n"], [M, N])
    c = torch.full(shape, float("nan"), dtype=torch.complex128, device="cuda") if c0 is None else c0.clone()
    d = Step(Operand.contiguous(("fixed", None), ["m", "k"], [M, K]),
             Operand.contiguous(("fixed", None), ["k", "n"], [K, N]), ["k"],
             Operand.contiguous(("fixed", None), lc, shape), alpha=alpha, beta=beta).desc
    a, b = a.contiguous(), b.contiguous()
    d.A, d.B, d.C = a.data_ptr(), b.data_ptr(), c.data_ptr()
    if tc:
        nbytes = int(lib.ptn_zcontract_work_bytes(ctypes.byref(d)))
        assert nbytes > 0, "the sizes must take the tensor-core path"
        work = torch.full((nbytes,), 0xff, dtype=torch.uint8, device="cuda")
        assert lib.ptn_zcontract_ws(ctypes.byref(d), work.data_ptr(), nbytes, _stream_ptr()) == 0
    else:
        assert lib.ptn_zcontract(ctypes.byref(d), _stream_ptr()) == 0
    torch.cuda.synchronize()
    return c.T if transposed else c


def _gauss(*shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, dtype=torch.complex128, device="cuda", generator=g)


def _sizes(*shape, seed, spread=10.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return _gauss(*shape, seed=seed + 1) * torch.exp(
        spread * torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g))


def _operands(kind):
    if kind == "small beside large":            # rows (1, r, 0, ...), columns (1, 1) and (0, 1)
        a = torch.zeros(1000, 40, dtype=torch.complex128, device="cuda")
        b = torch.zeros(40, 150, dtype=torch.complex128, device="cuda")
        a[:, 0] = 1
        a[:, 1] = torch.tensor([1e-3, 1e-12, 1e-18, 1e-30, 1e-200], dtype=torch.complex128, device="cuda").repeat(200)
        b[0, ::2] = 1
        b[1] = 1
    elif kind == "one large column":
        a, b = _gauss(8192, 16, seed=1), _gauss(16, 64, seed=2)
        a[:, 0] *= 1e10
        b[0, 5] = 0
    elif kind == "large at zeros":              # rows of zeros in one operand, the other one large there
        a, b = _gauss(777, 70, seed=3), _gauss(70, 129, seed=4)     # (edges of tiles, K steps and chunks)
        b[::3] = 0
        a[:, ::3] *= 1e20
        a[5, ::3] = 0
    elif kind == "identity part":               # a graded vector against (identity, dense) columns
        a = _gauss(2000, 64, seed=5) * torch.exp(-0.4 * torch.arange(64, dtype=torch.float64, device="cuda"))
        a *= torch.exp(-0.01 * torch.arange(2000, dtype=torch.float64, device="cuda"))[:, None]
        b = _gauss(64, 2, 64, seed=6)
        b[:, 0] = torch.eye(64, device="cuda")
        b = b.reshape(64, 128)
    elif kind == "all sizes":
        a, b = _sizes(1000, 90, seed=7), _sizes(90, 77, seed=8)
    elif kind == "all sizes, split":
        a, b = _sizes(200, 2500, seed=9), _sizes(2500, 45, seed=10)
    elif kind == "few of all sizes":            # some tiles in FP64, some rows within others
        a, b = _gauss(1500, 60, seed=11), _gauss(60, 100, seed=12)
        a[100:160] = _sizes(60, 60, seed=13)
        b[:, 70:] = torch.zeros_like(b[:, 70:])
        b[torch.arange(30) * 2, torch.arange(70, 100)] = 3.0 - 1j
    elif kind == "scattered":                   # a few to a warp, more than a CTA lists
        a = _sizes(20000, 16, seed=15, spread=1.5)
        b = torch.eye(16, dtype=torch.complex128, device="cuda").repeat(1, 4) * (0.7 - 0.2j)
    else:                                       # one entry to a column, and rows of every size
        a = _sizes(4097, 64, seed=14, spread=3.0)
        b = torch.eye(64, dtype=torch.complex128, device="cuda") * (0.3 + 0.7j)
    return a, b


# 128 x 32 tiles, K steps of 16, chunks of 64, 128 K and more to a range
@pytest.mark.parametrize("M,K,N", [(1100, 63, 127), (1101, 64, 128), (1100, 65, 129), (128, 255, 257), (33, 4113, 65),
                                   (90, 8100, 31), (65537, 10, 10), (8193, 17, 47)])
def test_sizes(M, K, N):
    a, b = _gauss(M, K, seed=M), _gauss(K, N, seed=N)
    tol = K * 2.0 ** -49 * (a.abs() @ b.abs())
    for x, y, t in ((a, b, tol), (b.T, a.T, tol.T)):
        assert bool(((_contract(x, y, True) - _contract(x, y, False)).abs() <= t).all())


@pytest.mark.parametrize("M,K,N", [(400, 96, 160), (300, 2500, 40)])
def test_not_finite_and_far_magnitudes(M, K, N):
    """NaN and infinities reach the outputs that they reach in the FP64 kernels; rows near
    the ends of the double range keep their relative accuracy."""
    a, b = _gauss(M, K, seed=40), _gauss(K, N, seed=41)
    a[5] = 0
    a[6] *= 1e-310
    a[7] *= 1e-200
    a[8] *= 1e200
    S = a.abs() @ b.abs()
    tc, plain = _contract(a, b, True), _contract(a, b, False)
    assert bool(((tc - plain).abs() <= K * 2.0 ** -49 * S + K * 2.0 ** -1070).all())
    assert not tc[5].any()
    a[3, 4], a[9, 2], b[8, 11] = complex("nan"), complex("inf"), complex("-inf")
    a[10, 8] = 0                                 # meets the infinity
    t, p = (torch.view_as_real(_contract(a, b, x)) for x in (True, False))
    assert torch.equal(torch.isnan(p), torch.isnan(t)) and torch.equal(torch.isinf(p), torch.isinf(t))
    assert not torch.isfinite(p[9]).any() and torch.isfinite(p[0, 0]).all()


@pytest.mark.parametrize("kind", ["small beside large", "one large column", "large at zeros", "identity part",
                                  "all sizes", "all sizes, split", "few of all sizes", "scattered", "one entry"])
@pytest.mark.parametrize("swapped", [False, True])
def test_every_output_is_held_to_its_own_terms(kind, swapped):
    a, b = _operands(kind)
    if swapped:
        a, b = b.T.contiguous(), a.T.contiguous()
    K = a.shape[1]
    plain = _contract(a, b, False)
    tol = K * 2.0 ** -49 * (a.abs() @ b.abs())
    for transposed in (False, True):
        tc = _contract(a, b, True, transposed)
        assert bool(((tc - plain).abs() <= tol).all()), float(((tc - plain).abs() / tol.clamp_min(1e-300)).max())
    # alpha and beta meet every output once, however it was summed
    c0 = _gauss(*plain.shape, seed=20)
    tc = _contract(a, b, True, alpha=0.5 - 2j, beta=-1.5, c0=c0)
    want = (0.5 - 2j) * plain - 1.5 * c0
    assert bool(((tc - want).abs() <= 4 * tol + 2.0 ** -49 * (plain.abs() + c0.abs())).all())


def test_hamiltonian_channels_of_unlike_size():
    """The TTNO product and the environment after it, the two that add the identity and
    the block-Hamiltonian channel in one sum, with block Hamiltonians 10^6 times the
    couplings: the 2-norm error of the result stays at FP64 rounding (sqrt(K) 2^-53 for
    the longer sum of K = 320, 2e-15; five times that here)."""
    chi, w, d, big = 64, 5, 2, 1e6
    scale = torch.tensor([1.0, big, 1.0, 1.0, 1.0], dtype=torch.float64, device="cuda")
    t = _gauss(4 * chi * chi, d, w, seed=30) * scale
    W = torch.zeros(d, w, w, w, d, dtype=torch.complex128, device="cuda")       # (s, i, k, l, t)
    one = torch.eye(2, dtype=torch.complex128, device="cuda")
    for i, k, l in ((1, 0, 0), (0, 1, 0), (0, 0, 1)):
        W[:, i, k, l] += one
    ops = _gauss(3, d, d, seed=31)
    for p in range(3):
        W[:, 2 + p, 0, 0] += ops[p]
        W[:, 0, 2 + p, 0] += ops[p]
        W[:, 0, 0, 2 + p] += ops[p]
    E = _gauss(chi, w, chi, seed=32) * scale[:, None] / chi ** 0.5
    E[:, 0] = torch.eye(chi, device="cuda")
    out = []
    for tc in (True, False):
        u = _contract(t.reshape(-1, d * w), W.reshape(d * w, -1), tc)              # (c, b), (k, l, t)
        u = u.reshape(4 * chi, chi, w, w * d).permute(0, 3, 1, 2).reshape(-1, chi * w)
        out.append(_contract(u, E.reshape(chi * w, chi), tc))
    assert float((out[0] - out[1]).norm() / out[1].norm()) <= 1e-14
