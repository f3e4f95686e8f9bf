"""What a tree-tensor-network time evolution spends its time on, as cases that can be timed and compared.

Each case is one pass through a public entry point of ``pytreenet_gb300`` on seeded inputs:

* ``step``     one ``run_one_time_step`` of ``FirstOrderOneSiteTDVP`` (and <Z_i> of every site where the case says so);
* ``site``     the update of one site, exp(-i dt H_eff) x (``DeviceNetwork.evolve_site``);
* ``env``      one environment update (``SandwichCache.update_tree_cache``);
* ``bond``     the backward evolution of a bond matrix (``effective_bond_evolution`` on device tensors);
* ``hop``      the orthogonality centre moved to a neighbour and back (``DeviceNetwork.move_orth_center``);
* ``pair``     a two-site update of a neighbouring pair and the update back (``DeviceNetwork.evolve_two_site``);
* ``observe``  <Z_i> of every site in one call (``DeviceNetwork.expect_many``);
* ``grad``     value and gradient of <Z_root> after a step (``OneSiteTDVPAdjoint.expectation_and_gradient``).

The states are as a time evolution meets them: isometric site tensors toward the orthogonality centre, bonds no larger
than the subtree below them can carry, Heisenberg (TTNO bond 5) or transverse-field Ising (TTNO bond 3) Hamiltonians
with random fields.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import pytreenet_gb300 as ptn
from pytreenet_gb300.engine import DeviceNetwork

CDT = torch.complex128
DT = 0.01
TOL = 1e-10
DEPTH = 7            # Krylov vectors of a local update at this step and tolerance (5 to 9 are seen)
X = np.array([[0, 1], [1, 0]], dtype=complex)
Y = np.array([[0, -1j], [1j, 0]], dtype=complex)
Z = np.diag([1.0, -1.0]).astype(complex)
BOND = {"heisenberg": 5, "ising": 3}


def listed() -> list[dict]:
    return [
        # a small tree followed in real time with every <Z_i> after each step: all launches and host calls
        {"name": "step_binary15_chi8", "kind": "step", "tree": "binary", "sites": 15, "chi": 8, "model": "ising",
         "precision": "plain", "observe": True},
        # the benchmark workload: a sweep of the 61-site T-tree at bond 256 on the tensor cores
        {"name": "step_ttree61_chi256_mixed", "kind": "step", "tree": "ttree", "sites": 61, "chi": 256,
         "model": "heisenberg", "precision": "mixed", "observe": False},
        # a site of a small tree with an odd bond dimension, the default precision
        {"name": "site_3legs_chi13", "kind": "site", "legs": 3, "chi": 13, "model": "ising", "precision": "plain"},
        # a branching site in complex128, the size a gradient or a two-site run works at
        {"name": "site_3legs_chi64", "kind": "site", "legs": 3, "chi": 64, "model": "heisenberg",
         "precision": "plain"},
        # an arm site at the benchmark's bond on the tensor cores: 57 of a sweep's 61 site updates
        {"name": "site_2legs_chi256_mixed", "kind": "site", "legs": 2, "chi": 256, "model": "heisenberg",
         "precision": "mixed"},
        # a branching site on the tensor cores, where the sweep's arithmetic is
        {"name": "site_3legs_chi128_mixed", "kind": "site", "legs": 3, "chi": 128, "model": "heisenberg",
         "precision": "mixed"},
        # an environment past a branching site, bond dimension no multiple of anything
        {"name": "env_3legs_chi90", "kind": "env", "legs": 3, "chi": 90, "model": "heisenberg",
         "precision": "plain"},
        # the link update of one-site TDVP
        {"name": "bond_chi128", "kind": "bond", "chi": 128, "model": "heisenberg"},
        # the QR splits of an arm at the benchmark's bond, there and back
        {"name": "hop_2legs_chi256", "kind": "hop", "legs": 2, "chi": 256, "precision": "plain"},
        # a two-site update (merge, exponential, truncated SVD) at the bond cap of the two-site workload
        {"name": "pair_2legs_chi64", "kind": "pair", "legs": 2, "chi": 64, "model": "heisenberg",
         "precision": "plain"},
        # a measurement of every site of the 61-site tree
        {"name": "observe_ttree61_chi64", "kind": "observe", "sites": 61, "chi": 64},
        # the backward direction: a step recomputed and differentiated
        {"name": "grad_binary15_chi16", "kind": "grad", "sites": 15, "chi": 16, "precision": "plain"},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["step", "site", "site", "site", "env", "env", "bond", "hop", "pair", "observe", "grad"])
    model = rng.choice(["heisenberg", "heisenberg", "ising"])
    precision = rng.choice(["plain", "plain", "mixed"])
    legs = rng.choice([2, 3])
    if kind == "step":
        if rng.random() < 0.5:
            return {"kind": "step", "tree": "binary", "sites": rng.choice([7, 15, 31]), "chi": _log(rng, 4, 14),
                    "model": model, "precision": "plain", "observe": True}
        return {"kind": "step", "tree": "ttree", "sites": 1 + 3 * rng.randint(3, 14), "chi": _log(rng, 24, 160),
                "model": model, "precision": "mixed", "observe": False}
    if kind == "site":
        top = {("plain", 2): 256, ("plain", 3): 64, ("mixed", 2): 256, ("mixed", 3): 128}[(precision, legs)]
        return {"kind": "site", "legs": legs, "chi": _log(rng, 8, top), "model": model, "precision": precision}
    if kind == "env":
        top = {2: 256, 3: 96 if precision == "plain" else 128}[legs]
        return {"kind": "env", "legs": legs, "chi": _log(rng, 8, top), "model": model, "precision": precision}
    if kind == "bond":
        return {"kind": "bond", "chi": _log(rng, 8, 256), "model": model}
    if kind == "hop":
        return {"kind": "hop", "legs": legs, "chi": _log(rng, 8, 256 if legs == 2 else 64), "precision": "plain"}
    if kind == "pair":
        return {"kind": "pair", "legs": legs, "chi": _log(rng, 4, 64 if legs == 2 else 16), "model": model,
                "precision": precision}
    if kind == "observe":
        return {"kind": "observe", "sites": 1 + 3 * rng.randint(3, 20), "chi": _log(rng, 8, 64)}
    return {"kind": "grad", "sites": rng.choice([7, 15]), "chi": _log(rng, 4, 16), "precision": "plain"}


# ----------------------------------------------------------------------------
# trees and their inputs
# ----------------------------------------------------------------------------
class Tree:
    """Sites (identifier, parent) in order, the root first, and the dimension of the bond above each."""

    def __init__(self, spec, bond):
        self.spec = spec
        self.ids = [n for n, _ in spec]
        self.parent = dict(spec)
        self.kids = {n: [c for c, p in spec if p == n] for n, _ in spec}
        self.bond = bond

    def nbrs(self, n):
        return ([self.parent[n]] if self.parent[n] is not None else []) + self.kids[n]

    def dim(self, a, b):
        return self.bond[b] if self.parent[b] == a else self.bond[a]

    def shape(self, n):
        return [self.dim(n, x) for x in self.nbrs(n)] + [2]


def _sizes(spec):
    size = {n: 1 for n, _ in spec}
    for n, p in reversed(spec):
        if p is not None:
            size[p] += size[n]
    return size


def _capped(spec, chi):
    """Bonds of dimension chi, capped by what the smaller side of the tree can carry."""
    size = _sizes(spec)
    return Tree(spec, {n: min(chi, 2 ** min(size[n], len(spec) - size[n], 40)) for n, p in spec if p is not None})


def _arms(legs, length):
    spec = [("c", None)]
    for a in range(legs):
        spec += [(f"a{a}_{k}", "c" if k == 0 else f"a{a}_{k - 1}") for k in range(length)]
    return spec


def _binary(sites):
    return [(f"s{i}", None if i == 0 else f"s{(i - 1) // 2}") for i in range(sites)]


def _tree(case) -> Tree:
    if case["kind"] in ("site", "env", "hop", "pair"):
        return _capped(_arms(case["legs"], max(2, math.ceil(math.log2(case["chi"])) + 1)), case["chi"])
    if case["kind"] == "observe" or case.get("tree") == "ttree":
        return _capped(_arms(3, (case["sites"] - 1) // 3), case["chi"])
    return _capped(_binary(case["sites"]), case["chi"])


def _gauss(shape, gen):
    return torch.view_as_complex(torch.randn(*shape, 2, dtype=torch.float64, device="cuda", generator=gen))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _tensors(tree, seed) -> dict:
    """Random site tensors on the GPU: isometries toward the root and a normalised root."""
    gen = _gen(seed)
    out = {}
    for n in tree.ids:
        shape = tree.shape(n)
        t = _gauss(shape, gen)
        if tree.parent[n] is not None:
            q, _ = torch.linalg.qr(t.reshape(shape[0], -1).T)          # rows: children and physical leg
            t = q.T.reshape(shape)
        else:
            t = t / t.norm()
        out[n] = t.contiguous()
    return out


def _operators(tree, model, seed) -> dict:
    """TTNO tensors (neighbours, out, in) of the nearest-neighbour model with random fields. A bond state is 0: nothing
    below the bond; 1: a whole term below it; 2 + a: the lower end of coupling a below it."""
    rng = np.random.default_rng(seed)
    pairs = [X, Y, Z] if model == "heisenberg" else [Z]
    field = Z if model == "heisenberg" else X
    w = BOND[model]
    out = {}
    for n in tree.ids:
        up, nk = tree.parent[n] is not None, len(tree.kids[n])
        W = np.zeros([w] * (nk + up) + [2, 2], dtype=complex)
        done = (1,) if up else ()
        if up:
            W[(0,) * (nk + 1)] = np.eye(2)
            for a, op in enumerate(pairs):
                W[(2 + a,) + (0,) * nk] = op
        W[done + (0,) * nk] += rng.uniform(-1.0, 1.0) * field
        for i in range(nk):
            at = [0] * nk
            at[i] = 1
            W[done + tuple(at)] += np.eye(2)
            for a, op in enumerate(pairs):
                at[i] = 2 + a
                W[done + tuple(at)] += op if model == "heisenberg" else -op
        out[n] = W
    return out


def _network(tree, tensors, cls):
    """The tensors as a TTNS or TTNO, built node by node."""
    ttn = cls()
    hung = {n: 0 for n in tree.ids}
    for n, p in tree.spec:
        t = tensors[n]
        t = t.cpu().numpy() if isinstance(t, torch.Tensor) else t
        if p is None:
            ttn.add_root(n, t)
        else:
            ttn.add_child_to_parent(n, t, 0, p, hung[p] + (tree.parent[p] is not None))
            hung[p] += 1
    return ttn


def _state(tree, tensors):
    psi = _network(tree, tensors, ptn.TTNS)
    psi.orthogonality_center_id = tree.ids[0]
    return psi


def _bond_inputs(case, seed):
    """A bond matrix and the environments of its two ends: identity, block Hamiltonian, coupled operators."""
    gen, chi, w = _gen(seed), case["chi"], BOND[case["model"]]

    def hermitian(norm):
        h = _gauss((chi, chi), gen)
        h = h + h.conj().T
        return h * (norm / (2.0 * math.sqrt(2.0 * chi)))
    ends = []
    for k in range(2):
        ops = [torch.eye(chi, dtype=CDT, device="cuda"), hermitian(10.0)]
        ops = (ops if k == 0 else ops[::-1]) + [hermitian(1.0) for _ in range(w - 2)]
        ends.append(torch.stack([o.T for o in ops], dim=1).contiguous())      # (ket, ham, bra)
    r = _gauss((chi, chi), gen)
    return (r / r.norm()).contiguous(), ends[0], ends[1]


# ----------------------------------------------------------------------------
# the passes
# ----------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "bond":
        r, up, down = _bond_inputs(case, seed)
        node = ptn.Node("bond")
        node.parent, node.children = "up", ["down"]
        envs = ptn.PartialTreeCachDict()
        envs.add_entry("up", "down", up)
        envs.add_entry("down", "up", down)
        return {"case": case, "r": r, "node": node, "envs": envs}
    tree = _tree(case)
    s = {"case": case, "tree": tree}
    psi = _state(tree, _tensors(tree, seed))
    if kind in ("hop", "observe"):
        s["net"] = DeviceNetwork(psi, None, precision=case.get("precision", "plain"))
        s["ops"] = [{n: Z} for n in tree.ids]
        return s
    model = case.get("model", "ising")
    ham = _network(tree, _operators(tree, model, seed), ptn.TTNO)
    if kind == "grad":
        s["adj"] = ptn.OneSiteTDVPAdjoint(psi, ham, 2 * DT, 1, krylov_tol=1e-12, normalise=True,
                                          precision=case["precision"])
    elif kind == "step":
        s["tdvp"] = ptn.FirstOrderOneSiteTDVP(psi, ham, DT, 100 * DT, {}, precision=case["precision"],
                                              config=ptn.TDVPConfig(time_evo_mode=ptn.TimeEvoMode.KRYLOV),
                                              solver_options={"krylov_tol": TOL})
        s["ops"] = [{n: Z} for n in tree.ids]
    else:
        s["cache"] = ptn.SandwichCache.init_cache_but_one(psi, ham, "c", precision=case["precision"])
        s["svd"] = ptn.SVDParameters(max_bond_dim=case["chi"], rel_tol=1e-10, total_tol=1e-10)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "bond":
        return ptn.effective_bond_evolution(s["r"], s["node"], DT, s["envs"], mode=ptn.TimeEvoMode.KRYLOV,
                                            forward=ptn.EvoDirection.BACKWARD, krylov_tol=TOL)
    if kind == "step":
        s["tdvp"].run_one_time_step()
        net = s["tdvp"].net
        out = [net.t[n] for n in s["tree"].ids]
        if case["precision"] == "mixed":       # a snapshot in the 32 bits that the tensor-core products carry
            out = [t.to(torch.complex64) for t in out]
        return out + [net.expect_many(s["ops"])] if case["observe"] else out
    if kind == "site":
        net = s["cache"].net
        net.evolve_site("c", DT, -1j, TOL, None)
        return net.t["c"]
    if kind == "env":
        s["cache"].update_tree_cache("c", "a0_0")
        return s["cache"].net.env_buf("c", "a0_0")
    if kind == "hop":
        net = s["net"]
        net.move_orth_center("a0_0")
        net.move_orth_center("c")
        return [net.t["c"], net.t["a0_0"]]
    if kind == "pair":
        net = s["cache"].net
        there = net.evolve_two_site("c", "a0_0", DT, -1j, TOL, None, s["svd"])
        back = net.evolve_two_site("a0_0", "c", DT, -1j, TOL, None, s["svd"])
        return [net.t["c"], net.t["a0_0"], there, back]
    if kind == "observe":
        return s["net"].expect_many(s["ops"])
    value, g_ham, g_state = s["adj"].expectation_and_gradient({"s0": Z}, wrt_state=True)
    return [value] + [g_ham[n] for n in s["tree"].ids] + [g_state[n] for n in s["tree"].ids]


# ----------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------
def _macs(dims, w, close=True):
    """Complex multiply-adds of H_eff on a site with virtual legs ``dims`` (each environment in turn, the TTNO tensor in
    the middle); without ``close`` the last leg stays open."""
    legs = dims if close else dims[:-1]
    size, macs, half = 2 * math.prod(dims), 0, len(legs) // 2
    for i, d in enumerate(legs):
        macs += size * d * (w ** (i + 1 if i < half else len(dims) - i))
    return macs + size * 2 * w ** len(dims)


def work(case):
    kind = case["kind"]
    chi, w = case["chi"], BOND[case.get("model", "ising")]
    if kind == "bond":
        n = chi * chi
        return {"bytes": 16 * (2 * w * n + 2 * n), "flops": 8 * DEPTH * (2 * w * n * chi + 2 * DEPTH * n)}
    tree = _tree(case)
    c = tree.ids[0]
    size = {n: math.prod(tree.shape(n)) for n in tree.ids}
    env = sum(w * tree.dim("c", x) ** 2 for x in tree.nbrs("c")) if kind in ("site", "env", "pair") else 0
    if kind == "site":
        dims = tree.shape(c)[:-1]
        return {"bytes": 16 * (2 * size[c] + env),
                "flops": 8 * (DEPTH * _macs(dims, w) + 2 * DEPTH * DEPTH * size[c])}
    if kind == "env":
        dims = tree.shape(c)[:-1]
        d = dims[0]
        return {"bytes": 16 * (size[c] + env), "flops": 8 * (_macs(dims[1:] + [d], w, False) + size[c] * w * d)}
    if kind == "hop":
        d = tree.dim("c", "a0_0")
        n = size["c"] + size["a0_0"]
        return {"bytes": 16 * 2 * n, "flops": 8 * 3 * n * d}
    if kind == "pair":
        d = tree.dim("c", "a0_0")
        m, k = size["c"] // d, size["a0_0"] // d
        macs = DEPTH * m * k * (2 * w * chi + 8 * w * w) + 8 * min(m, k) ** 2 * max(m, k) + m * k * d
        return {"bytes": 16 * (2 * (size["c"] + size["a0_0"]) + env), "flops": 8 * 2 * macs}
    sites = sum(size.values())
    norms = sum(size[n] * max(tree.shape(n)) * (len(tree.shape(n)) - 1) for n in tree.ids)
    if kind == "observe":
        return {"bytes": 16 * sites, "flops": 8 * 2 * norms}
    macs = sum(DEPTH * _macs(tree.shape(n)[:-1], w) for n in tree.ids)
    macs += sum(DEPTH * 2 * w * d ** 3 for d in tree.bond.values())
    macs += sum((_macs(tree.shape(n)[:-1], w, False) + 3 * size[n] * max(tree.shape(n))) for n in tree.ids)
    if kind == "grad":
        return {"bytes": 16 * 3 * sites, "flops": 8 * 4 * macs}
    return {"bytes": 16 * 2 * sites, "flops": 8 * (macs + (2 * norms if case["observe"] else 0))}


# ----------------------------------------------------------------------------
# the same results from plain torch and numpy in 64 bits
# ----------------------------------------------------------------------------
def _envs(tree, tensors, ops) -> dict:
    """Environments (ket, ham, bra) of every site below the root toward its parent."""
    out = {}
    for n in reversed(tree.ids[1:]):
        out[n] = _env(tensors[n], ops[n], [None] + [out[c] for c in tree.kids[n]], 0)
    return out


def _apply(x, W, envs, open_leg=None):
    """H_eff x, or with a leg left open the sum before the bra tensor: the first environment, the TTNO tensor, the rest."""
    n = x.dim() - 1
    ket, ham, bra = "abcd"[:n], "ijkl"[:n], "mnop"[:n]
    T, legs = x, ket + "s"

    def fold(T, legs, k):
        new = legs.replace(ket[k], "").replace(ham[k], "") + ("" if ham[k] in legs else ham[k]) + bra[k]
        return torch.einsum(f"{legs},{ket[k]}{ham[k]}{bra[k]}->{new}", T, envs[k]), new
    if open_leg != 0:
        T, legs = fold(T, legs, 0)
    held = "".join(h for h in ham if h in legs)
    new = "".join(c for c in legs if c not in held + "s") + "".join(h for h in ham if h not in held) + "t"
    T, legs = torch.einsum(f"{legs},{ham}ts->{new}", T, W), new
    for k in range(1, n):
        if k != open_leg:
            T, legs = fold(T, legs, k)
    if open_leg is None:
        return torch.einsum(f"{legs}->{bra}t", T)
    return T, legs, (ket[open_leg], ham[open_leg], bra)


def _env(x, W, envs, toward):
    T, legs, (ket, ham, bra) = _apply(x, W, envs, open_leg=toward)
    return torch.einsum(f"{legs},{bra}t->{ket}{ham}{bra[toward]}", T, x.conj())


def _exp(x, act, factor):
    """exp(factor A) x by its Taylor series (|factor A| is about 1 here)."""
    total, term = x.clone(), x
    for k in range(1, 80):
        term = act(term) * (factor / k)
        total += term
        if float(term.norm()) < 1e-18 * float(total.norm()):
            break
    return total


def _qr(t, leg):
    """Q (t's legs) and R of t with ``leg`` as the column index, LAPACK's signs."""
    m = t.movedim(leg, -1)
    q, r = np.linalg.qr(m.reshape(-1, m.shape[-1]).cpu().numpy())
    q = torch.from_numpy(q).cuda().reshape(m.shape).movedim(-1, leg)
    return q.contiguous(), torch.from_numpy(r).cuda()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "grad"):
        return None
    if kind == "bond":
        r, up, down = _bond_inputs(case, seed)
        return _exp(r, lambda y: torch.einsum("bpc,cbq->pq", torch.einsum("abp,ac->bpc", up, y), down), 1j * DT)
    tree = _tree(case)
    t = _tensors(tree, seed)
    if kind == "hop":
        a, b = t["c"], t["a0_0"]
        a, r = _qr(a, 0)
        b = torch.einsum("na,abs->nbs", r, b)
        b, r = _qr(b, 0)
        return [torch.tensordot(r, a, dims=([1], [0])), b]
    if kind == "observe":
        return _all_z(tree, t)
    ops = {n: torch.from_numpy(W).cuda() for n, W in _operators(tree, case["model"], seed).items()}
    below = _envs(tree, t, ops)
    envs = [below[x] for x in tree.kids["c"]]
    if kind == "env":
        return _env(t["c"], ops["c"], envs, 0)
    if kind == "site":
        return _exp(t["c"], lambda y: _apply(y, ops["c"], envs), -1j * DT)
    # the pair: theta[rest of c, physical of c, child of a0_0, physical of a0_0]
    theta = torch.einsum("xms,xnt->msnt", t["c"].reshape(t["c"].shape[0], -1, 2), t["a0_0"])
    low = below["a0_1"]
    rest = t["c"].shape[1:-1]

    def act(y):
        # a0_0's side first (its TTNO leg toward c stays open), then c's
        y = torch.einsum("msnt,nkp->mstkp", y, low)
        y = torch.einsum("mstkp,bkut->msbpu", y, ops["a0_0"])
        if len(rest) == 1:
            y = torch.einsum("msbpu,mjq->sbpujq", y, envs[1])
            return torch.einsum("sbpujq,bjvs->qvpu", y, ops["c"])
        y = y.reshape(rest + y.shape[1:])
        y = torch.einsum("mnsbpu,mjq->nsbpujq", y, envs[1])
        y = torch.einsum("nsbpujq,bjlvs->npuqlv", y, ops["c"])
        y = torch.einsum("npuqlv,nlr->qrvpu", y, envs[2])
        return y.reshape((-1,) + y.shape[2:])
    kept = []
    for _ in range(2):
        theta = _exp(theta, act, -1j * DT)
        m = theta.reshape(theta.shape[0] * 2, -1)
        u, s, v = np.linalg.svd(m.cpu().numpy(), full_matrices=False)
        r = min(case["chi"], int(np.sum(s > max(1e-10 * s[0], 1e-10))))
        kept.append(s[:r])
        theta = torch.from_numpy((u[:, :r] * s[:r]) @ v[:r]).cuda().reshape(theta.shape)
    return [None, None, kept[0], kept[1]]


def _all_z(tree, t):
    """<Z_i> of every site of a state that is isometric toward the root: the reduced density of each bond is carried
    from the root outward."""
    z = torch.from_numpy(Z).cuda()
    out = {}

    def down(n, rho):
        x = t[n]
        if rho is None:
            y = x
        else:
            y = torch.tensordot(rho, x, dims=([0], [0]))            # (bra of the parent's bond, rest...)
        flat = x.conj().reshape(-1, 2)
        out[n] = torch.einsum("rs,rt,ts->", y.reshape(-1, 2), flat, z)
        up = tree.parent[n] is not None
        for i, c in enumerate(tree.kids[n]):
            a, b = (v.movedim(i + up, 0).reshape(x.shape[i + up], -1) for v in (y, x.conj()))
            down(c, a @ b.T)
    down(tree.ids[0], None)
    return torch.stack([out[n] for n in tree.ids])
