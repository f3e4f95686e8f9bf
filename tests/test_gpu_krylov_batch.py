"""The Krylov exponential driven by ``ptn_krylov_batch`` against the same solve one
step at a time from the host (a plan whose run() is replaced takes that path):
depths, stops and results. The two form exp(z T) e_1 of the same projection in
different ways (Taylor steps, eigenvectors): 1e-14 of the vector's norm each."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _net(precision):
    import pytreenet_gb300 as ptn
    from pytreenet_gb300.workloads import t_tree_heisenberg, t_tree_state
    psi, _, _ = t_tree_state(arm_len=3, chi=8, seed=2)
    ham, _ = t_tree_heisenberg(psi, seed=3)
    cache = ptn.SandwichCache(psi, ham, precision=precision)
    cache.net.canonical_form("root")
    cache.net.normalise_center()
    cache.net.init_cache_but_one("root")
    return cache.net


@pytest.mark.parametrize("precision", ["plain", "mixed"])
@pytest.mark.parametrize("dt,tol,maxdim", [(0.01, 1e-10, None), (0.4, 1e-10, None), (2.0, 1e-12, None), (0.4, 0.0, 9),
                                           (0.4, 1e-10, 5), (0.02, 1e-6, 1)])
def test_krylov_batch_matches_the_loop(precision, dt, tol, maxdim):
    from pytreenet_gb300.engine import KrylovSolver, Workspace
    net = _net(precision)
    p = net.heff_plan("root")
    x = net.t["root"].clone()
    out, depth = [], []
    for native in (True, False):
        if not native:
            p.run = p.run                               # an instance attribute: the loop runs it
        solver = KrylovSolver(net.ws)                   # no memory of earlier depths
        y = torch.empty_like(x)
        for _ in range(2):                              # from 4 speculative steps, then from the depth found
            basis = {}
            net._held(p, lambda: solver.expm(x, net._plan_apply(p), dt, -1j, tol, maxdim, out=y,
                                             tridiagonal=net.levels > 0, basis=basis))
        out.append(y)
        depth.append((list(solver.depths), basis["m"], basis["beta0"], tuple(basis["Q"].shape)))
    del p.run
    assert depth[0] == depth[1]
    scale = max(1.0, 20.0 * dt)                          # |z H| of this Hamiltonian is below 20 dt
    assert float((out[0] - out[1]).norm()) <= 4e-14 * scale * float(x.norm())
    if maxdim is None and precision == "plain":
        assert abs(float(out[0].norm()) - float(x.norm())) < 1e-9


def test_krylov_batch_zero_vector_and_counts():
    net = _net("plain")
    p = net.heff_plan("root")
    net.krylov.expm(torch.zeros_like(net.t["root"]), net._plan_apply(p), 0.1, -1j, out=(z := net.t["root"].clone()))
    assert float(z.abs().max()) == 0.0
    f0 = net.flops
    net.evolve_site("root", 0.01, -1j, 1e-10, None)
    assert (net.flops - f0) % p.flops == 0 and net.flops - f0 >= p.flops * net.krylov.depths[-1]
    x = net.t["root"]
    x.view(-1)[3] = complex("nan")
    from pytreenet_gb300._lib import PtnError
    with pytest.raises(PtnError):
        net.evolve_site("root", 0.01, -1j, 1e-10, None)


def test_krylov_batch_depth_beyond_one_block():
    """More than 64 vectors: the combination runs in blocks."""
    net = _net("plain")
    p = net.heff_plan("root")
    x = net.t["root"].clone()
    y = torch.empty_like(x)
    net.krylov.expm(x, net._plan_apply(p), 6.0, -1j, 1e-10, None, out=y)
    assert net.krylov.depths[-1] > 64
    z = x.clone()
    for _ in range(24):
        net.krylov.expm(z, net._plan_apply(p), 0.25, -1j, 1e-13, None, out=z)
    assert float((y - z).norm()) < 1e-8
    assert np.isfinite(float(y.norm()))
