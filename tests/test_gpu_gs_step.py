"""The Gram-Schmidt step of the Krylov exponential at the edges of its launch shapes
(one CTA up to 128 entries, up to 152 CTAs with w in shared memory, one launch per
pass above 152 x 12800 entries, one kernel per operation above 16 vectors) against
torch in FP64. Both sides sum at most n products of unit vectors: 2 n 2^-53."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nq", [(1, 1), (31, 3), (128, 2), (129, 5), (257, 16), (19456, 7), (19457, 9), (50000, 17),
                                  (1945600, 2), (1945601, 3), (1945601, 12), (4394, 11), (4394, 13), (70001, 15)])
@pytest.mark.parametrize("with_next", [True, False])
def test_gs_step_sizes(n, nq, with_next):
    from pytreenet_gb300 import _lib
    from pytreenet_gb300.engine import _stream_ptr
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(n + nq)
    Q = torch.randn(nq, n, dtype=torch.complex128, device="cuda", generator=g)
    Q /= Q.norm(dim=1, keepdim=True)
    w0 = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)
    w0 /= w0.norm()
    # scratch that anything may have been left in
    part = torch.full((int(lib.ptn_krylov_partials(n)),), complex(1.0, 2.0 ** -1042), dtype=torch.complex128, device="cuda")
    results = []
    for _ in range(2):
        w = w0.clone()
        h = torch.full((2 * nq,), float("nan"), dtype=torch.complex128, device="cuda")
        norms = torch.full((2,), float("nan"), dtype=torch.float64, device="cuda")
        nxt = torch.full((n,), float("nan"), dtype=torch.complex128, device="cuda")
        assert lib.ptn_krylov_gs_step(Q.data_ptr(), n, nq, w.data_ptr(), n, h.data_ptr(), part.data_ptr(),
                                      norms.data_ptr(), nxt.data_ptr() if with_next else None, _stream_ptr()) == 0
        results.append((w, h, norms, nxt))
    torch.cuda.synchronize()
    for a, b in zip(results[0][:3], results[1][:3]):
        assert torch.equal(a, b)                        # the same bits on every run
    w, h, norms, nxt = results[0]
    h1 = Q.conj() @ w0
    w1 = w0 - h1 @ Q
    h2 = Q.conj() @ w1
    w2 = w1 - h2 @ Q
    tol = 2.0 ** -52 * n * (nq + 2) + 2.0 ** -50
    assert float((h[:nq] - h1).abs().max()) < tol and float((h[nq:] - h2).abs().max()) < tol * (nq + 1)
    assert float((w - w2).norm()) < tol * (nq + 1)
    assert abs(float(norms[0]) - 1.0) < tol and abs(float(norms[1]) - float(w.norm())) < tol
    if with_next and float(norms[1]) > 0:
        assert float((nxt - w / norms[1]).norm()) < 2.0 ** -50
