"""The Krylov exponential from native code at long time steps, |z H| from 1 to 1e8: the
series that forms exp(z T) e_1 of the projection is for short ones, the others go through
eigendecompositions. Against the dense exponential of the effective Hamiltonian: the
phases of its eigenvalues are known to eps |z H|, times 64 for the sums, beside the
Krylov tolerance 1e-10 (a factor of ten for the estimate that stops the solve)."""
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _net(chi, arm_len):
    import pytreenet_gb300 as ptn
    from pytreenet_gb300.workloads import t_tree_heisenberg, t_tree_state
    psi, _, _ = t_tree_state(arm_len=arm_len, chi=chi, seed=2)
    ham, _ = t_tree_heisenberg(psi, seed=3)
    cache = ptn.SandwichCache(psi, ham, precision="plain")
    cache.net.canonical_form("root")
    cache.net.normalise_center()
    cache.net.init_cache_but_one("root")
    return cache.net


def _solve(net, x, dt, native, maxdim=None, factor=-1j, tol=1e-10):
    from pytreenet_gb300.engine import KrylovSolver
    p = net.heff_plan("root")
    if not native:
        p.run = p.run                               # an instance attribute: the loop runs it
    try:
        solver, y = KrylovSolver(net.ws), torch.empty_like(x)
        best = np.inf
        for _ in range(3):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            solver.expm(x, net._plan_apply(p), dt, factor, tol, maxdim, out=y)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t0)
        return y, solver.depths[-1], best
    finally:
        vars(p).pop("run", None)


@pytest.mark.parametrize("size", [1.0, 1e2, 1e4, 1e8])
@pytest.mark.parametrize("factor", [-1j, 1j])
def test_long_steps_against_the_dense_exponential(size, factor):
    net = _net(2, 2)
    p, x = net.heff_plan("root"), net.t["root"].clone()
    n = x.numel()
    H = np.zeros((n, n), dtype=complex)
    for i in range(n):
        e = torch.zeros(n, dtype=torch.complex128, device="cuda")
        e[i] = 1.0
        y = torch.empty_like(e)
        p.run(e.data_ptr(), y.data_ptr())
        H[:, i] = y.cpu().numpy()
    ev, V = np.linalg.eigh(0.5 * (H + H.conj().T))
    dt = size / np.abs(ev).max()
    ref = V @ (np.exp(factor * dt * ev) * (V.conj().T @ x.cpu().numpy().reshape(-1)))
    y, _, _ = _solve(net, x, dt, True, factor=factor)
    assert np.linalg.norm(y.cpu().numpy().reshape(-1) - ref) <= 64 * 2.3e-16 * size + 1e-9


@pytest.mark.parametrize("dt,maxdim,tol", [(5.0, 64, 1e-10), (20.0, 64, 1e-10), (0.4, 64, 0.0)])
def test_long_steps_take_no_longer_than_the_loop(dt, maxdim, tol):
    """The same depth and result, and no more time than one step at a time with an
    eigendecomposition each (half as much again, and 5 ms, for the machine)."""
    net = _net(8, 3)
    x = net.t["root"].clone()
    a, da, ta = _solve(net, x, dt, True, maxdim, tol=tol)
    b, db, tb = _solve(net, x, dt, False, maxdim, tol=tol)
    assert da == db
    assert float((a - b).norm()) <= 4e-14 * max(1.0, 20.0 * dt)
    assert ta <= 1.5 * tb + 5e-3


def test_no_krylov_vector_is_refused():
    net = _net(2, 2)
    with pytest.raises((ValueError, IndexError)):
        _solve(net, net.t["root"].clone(), 0.1, True, maxdim=0)
