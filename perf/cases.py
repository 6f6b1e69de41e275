"""Measured cases of the sweep path: what a user's DMRG or TDVP program runs per region,
and two whole calls.

Every case goes through the package's public entry points on states and operators made
here from the seed: random tensor networks in the sweep's gauge (isometries toward the
region, bond dimensions capped as in a run) under the operators of `models`.  Outputs do
not depend on the gauge of a bond (a product of site tensors, not the site tensors
themselves), so two correct programs agree on them.  `exact` restates each block in plain
torch at 64 bits (the energies of the whole calls have no such closed form).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import networksolvers_gb300 as ns
from networksolvers_gb300 import _native, batch, models
from networksolvers_gb300.itensors import DTensor, Index, contract, factorize
from networksolvers_gb300.network import LinearMap, ProjTTN, from_network
from networksolvers_gb300.sweep import (ApplyExpProblem, EigsolveProblem, RegionIterator, eigsolve_solver,
                                        exponentiate_solver, region_iterator_action, region_step, updater_applyexp,
                                        updater_eigsolve)


def listed():
    return [
        # the reference's own N=20 Heisenberg run: one fused region step at its bond dimension
        dict(name="region_c1", kind="region", chi_l=64, chi_r=64, chi_c=64, maxdim=64, cutoff=1e-10, model="heisenberg",
             direction=0, precision="fp64"),
        # a served XXZ request in the split form, ragged bonds, right-to-left pass
        dict(name="region_xxz", kind="region", chi_l=229, chi_r=187, chi_c=241, maxdim=256, cutoff=1e-10, model="xxz",
             direction=1, precision="ozaki"),
        # the local eigensolve of the N=100 run at its largest bond dimension
        dict(name="eigsolve_split", kind="eigsolve", chi_l=1024, chi_r=1024, model="heisenberg", precision="ozaki"),
        # the same in the plain form, on a J1-J2 chain (operator bond 8)
        dict(name="eigsolve_plain", kind="eigsolve", chi_l=259, chi_r=231, model="j1j2", precision="fp64"),
        # the environment update after a region of the N=100 run (a bond dimension it passes through)
        dict(name="environment", kind="environment", chi_l=843, chi_r=590, model="heisenberg", precision="ozaki"),
        # a two-site TDVP step on the binary tree at the small bond dimensions of a quench
        dict(name="tdvp_tree", kind="tdvp", graph="tree", depth=4, chi=6, dt=0.05, cutoff=1e-9, precision="fp64"),
        # a two-site TDVP step of a chain quench, complex, split form
        dict(name="tdvp_chain", kind="tdvp", graph="chain", depth=18, chi=128, dt=0.05, cutoff=1e-9,
             precision="ozaki"),
        # the truncated factorization of a converged two-site tensor (N=100 run: bonds 475)
        dict(name="factorize_square", kind="factorize", rows=950, cols=950, keep=475, complex=False,
             precision="ozaki"),
        # and of a sweep that raises the bond dimension: tall, every state kept, weights down to 1e-12
        dict(name="factorize_tall", kind="factorize", rows=2048, cols=1024, keep=1024, complex=False,
             precision="ozaki"),
        # one region of the general driver with the density-matrix expansion, converged N=100 shape
        dict(name="expand", kind="expand", chi=475, maxdim=1024, precision="ozaki"),
        # the whole reference run: N=20 Heisenberg, 5 sweeps, maxdim 64, through `dmrg`
        dict(name="dmrg_n20", kind="dmrg", n=20, chi0=10, maxdim=64, nsweeps=5, cutoff=1e-10, precision="fp64"),
        # a batch of independent J1-J2 chains of uneven length and bond dimension on a solve pool
        dict(name="batch", kind="batch", chains=8, nmin=16, nmax=32, maxdim=64, nsweeps=2, workers=8,
             precision="ozaki"),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    """One more case: the kinds weighted by how often a sweep runs them, sizes over the
    logarithm of their range."""
    kind = rng.choice(["region", "region", "region", "eigsolve", "eigsolve", "environment", "tdvp", "tdvp", "factorize",
                       "factorize", "factorize", "expand", "dmrg", "batch"])
    split = rng.random() < 0.6
    precision = "ozaki" if split else "fp64"
    model = rng.choice(["heisenberg", "xxz", "j1j2"])
    if kind == "region":
        a, b = _log(rng, 16, 256), _log(rng, 16, 256)
        c = min(2 * a, 2 * b, _log(rng, 16, 256))
        return dict(kind=kind, chi_l=a, chi_r=b, chi_c=c, maxdim=min(256, c + c // 8), cutoff=1e-10, model=model,
                    direction=rng.randrange(2), precision=precision)
    if kind == "eigsolve":
        top = 1024 if split else 300
        a, b = _log(rng, 16, top), _log(rng, 16, top)
        return dict(kind=kind, chi_l=a, chi_r=b, model=model if max(a, b) < 800 else "heisenberg", precision=precision)
    if kind == "environment":
        top = 1024 if split else 300
        a = _log(rng, 16, top)
        return dict(kind=kind, chi_l=a, chi_r=min(2 * a, _log(rng, 16, top)), model=model, precision=precision)
    if kind == "tdvp":
        if rng.random() < 0.5:
            return dict(kind=kind, graph="tree", depth=rng.choice([3, 4, 5]), chi=_log(rng, 2, 10), dt=0.05,
                        cutoff=1e-9, precision=precision)
        return dict(kind=kind, graph="chain", depth=18, chi=_log(rng, 8, 160), dt=rng.choice([0.02, 0.05]),
                    cutoff=1e-9, precision=precision)
    if kind == "factorize":
        cplx = rng.random() < 0.25
        n = _log(rng, 24, 1024 if split and not cplx else 512)
        shape = rng.choice(["square", "tall", "wide"])
        m = n if shape == "square" else _log(rng, n, 2 * n)
        if shape == "wide":
            m, n = n, m
        keep = min(m, n) if shape == "tall" else max(8, int(min(m, n) * rng.uniform(0.3, 0.7)))
        return dict(kind=kind, rows=m, cols=n, keep=keep, complex=cplx, precision=precision)
    if kind == "expand":
        chi = _log(rng, 48, 475)
        return dict(kind=kind, chi=chi, maxdim=int(chi * rng.uniform(1.3, 2.2)), precision="ozaki")
    if kind == "dmrg":
        return dict(kind=kind, n=rng.randrange(10, 21), chi0=rng.choice([4, 8, 10]), maxdim=rng.choice([24, 32, 64]),
                    nsweeps=rng.randrange(2, 5), cutoff=1e-10, precision=precision)
    return dict(kind=kind, chains=rng.randrange(4, 9), nmin=12, nmax=rng.randrange(16, 33),
                maxdim=rng.choice([32, 64]), nsweeps=2, workers=8, precision=precision)


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------

_contexts = {}


def _context(precision):
    """One context per precision form, as a program keeps."""
    if precision not in _contexts:
        _contexts[precision] = _native.Context(0, precision=precision)
    return _contexts[precision]


def _operator(model, n, rng):
    if model == "xxz":
        return models.xxz_chain(n, float(rng.uniform(0.2, 1.8)))
    if model == "j1j2":
        return models.j1j2_chain(n, float(rng.uniform(0.1, 0.5)))
    return models.heisenberg_chain(n)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _randn(shape, g, cplx=False):
    x = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
    return torch.complex(x, torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)) if cplx else x


def _sizes(graph, cap):
    """Bond dimension of every edge: 2^(sites on the smaller side), at most cap(edge)."""
    out = {}
    for (u, v) in graph.edges:
        seen, stack = {u}, [u]
        while stack:
            x = stack.pop()
            for y in graph.neighbors(x):
                if y not in seen and not (x == u and y == v):
                    seen.add(y)
                    stack.append(y)
        side = min(len(seen), len(graph.vertices) - len(seen))
        out[(u, v)] = min(2 ** min(side, 30), cap((u, v)))
    return out


def _state(graph, dims, root, g, cplx=False):
    """Random network in the gauge with orthogonality centre `root`: every other tensor an
    isometry toward it, the centre normalised."""
    legs = models.random_state(graph, 1).legs
    toward, order = {root: None}, [root]
    for v in order:
        for u in graph.neighbors(v):
            if u not in toward:
                toward[u] = v
                order.append(u)
    tensors = {}
    for v in graph.vertices:
        size = {l: (2 if l[0] == "s" else dims[l[1]]) for l in legs[v]}
        if v == root:
            t = _randn([size[l] for l in legs[v]], g, cplx)
            tensors[v] = (t / t.norm()).cpu().numpy()
            continue
        up = ("l", graph.edge_key(v, toward[v]))
        rest = [l for l in legs[v] if l != up]
        rows = math.prod(size[l] for l in rest)
        q = torch.linalg.qr(_randn([rows, size[up]], g, cplx))[0].reshape([size[l] for l in rest] + [size[up]])
        tensors[v] = q.permute([(rest + [up]).index(l) for l in legs[v]]).cpu().numpy()
    return models.Network(graph, tensors, legs, np.complex128 if cplx else np.float64,
                          {"kind": "state", "ortho_region": [root]})


def _dot(a, la, b, lb):
    """Contraction of two labelled torch tensors over their shared labels."""
    k = [x for x in la if x in lb]
    t = torch.tensordot(a, b, dims=([la.index(x) for x in k], [lb.index(x) for x in k]))
    return t, [x for x in la if x not in k] + [x for x in lb if x not in k]


def _site(net, v, dtype):
    return torch.from_numpy(np.ascontiguousarray(net.tensors[v])).to("cuda", dtype), list(net.legs[v])


def _bra(names):
    return [("b", x[1]) if x[0] == "l" else ("sp", x[1]) if x[0] == "s" else x for x in names]


def _env(H, psi, u, v, dtype):
    """Environment of the vertices on u's side of edge (u, v), as [bra, operator, ket]."""
    A, la = _site(psi, u, dtype)
    T, lt = A, la
    for w in psi.graph.neighbors(u):
        if w != v:
            e = psi.graph.edge_key(w, u)
            T, lt = _dot(T, lt, _env(H, psi, w, u, dtype), [("b", e), ("w", e), ("l", e)])
    W, lw = _site(H, u, dtype)
    T, lt = _dot(T, lt, W, lw)
    T, lt = _dot(T, lt, A.conj(), _bra(la))
    e = psi.graph.edge_key(u, v)
    return T.permute([lt.index(x) for x in (("b", e), ("w", e), ("l", e))]).contiguous()


def _chain(case, seed):
    """(operator, state, left site, L, R) of a chain whose region (j, j+1) sits between bonds
    chi_l and chi_r, with the two environments as torch tensors."""
    left, right = math.ceil(math.log2(case["chi_l"])), math.ceil(math.log2(case["chi_r"]))
    j = left + 1
    graph = models.chain_graph(left + right + 2)
    rng = np.random.default_rng(seed)
    H = _operator(case["model"], len(graph.vertices), rng)
    mid = case.get("chi_c") or min(2 * case["chi_l"], 2 * case["chi_r"], max(case["chi_l"], case["chi_r"]))
    dims = _sizes(graph, lambda e: case["chi_l"] if e[0] < j else mid if e[0] == j else case["chi_r"])
    psi = _state(graph, dims, j, _gen(seed))
    L = _env(H, psi, j - 1, j, torch.float64)
    R = _env(H, psi, j + 2, j + 1, torch.float64)
    return H, psi, j, L, R


def _up(x, inds, ctx):
    return DTensor.from_numpy(x.cpu().numpy() if isinstance(x, torch.Tensor) else x, inds, ctx=ctx)


class _Fixed:
    """Fixed tensors of a region's effective Hamiltonian, in the order `optimal_map` takes."""

    def __init__(self, tensors):
        self.tensors = tensors

    def map_tensors(self):
        return self.tensors


def _prepare_chain_region(case, seed, ctx):
    H, psi, j, L, R = _chain(case, seed)
    W1, W2 = H.tensors[j], H.tensors[j + 1]
    a, b, c = Index(L.shape[0]), Index(R.shape[0]), Index(psi.tensors[j].shape[2])
    s1, s2 = Index(2), Index(2)
    w1, w2, w3 = Index(W1.shape[0]), Index(W1.shape[3]), Index(W2.shape[3])
    t = dict(L=_up(L, [a.prime(), w1, a], ctx), R=_up(R, [b.prime(), w3, b], ctx),
             W1=_up(W1, [w1, s1.prime(), s1, w2], ctx), W2=_up(W2, [w2, s2.prime(), s2, w3], ctx),
             psi1=_up(psi.tensors[j], [a, s1, c], ctx), psi2=_up(psi.tensors[j + 1], [c, s2, b], ctx))
    if case["kind"] == "eigsolve":
        t["x"] = t["psi1"] * t["psi2"]
    return t


def _tree_case(case, seed):
    """(operator, state, region) of a TDVP region at the middle of a chain or of the tree."""
    rng = np.random.default_rng(seed)
    h = float(rng.uniform(0.5, 1.5))
    if case["graph"] == "tree":
        graph, region = models.binary_tree_graph(case["depth"]), [1, 0]
    else:
        graph = models.chain_graph(case["depth"])
        region = [case["depth"] // 2, case["depth"] // 2 + 1]
    H = models.tfim_tree(graph, h=h).astype(np.complex128)
    psi = _state(graph, _sizes(graph, lambda e: case["chi"]), region[0], _gen(seed), cplx=True)
    return H, psi, region


def _expand_case(case, seed):
    k = math.ceil(math.log2(case["chi"]))
    graph = models.chain_graph(2 * k + 4)
    psi = _state(graph, _sizes(graph, lambda e: case["chi"]), k + 2, _gen(seed))
    return models.heisenberg_chain(len(graph.vertices)), psi, k + 2


def _matrix(case, seed):
    """A two-site tensor as a matrix with a graded spectrum: kept singular values down to
    10^-4.5 of the largest and the rest below 10^-7, or (keep = the narrow side) weights
    down to 10^-12.5, all kept."""
    m, n, k = case["rows"], case["cols"], case["keep"]
    r, g = min(m, n), _gen(seed)
    q1 = torch.linalg.qr(_randn([m, r], g, case["complex"]))[0]
    q2 = torch.linalg.qr(_randn([n, r], g, case["complex"]))[0]
    i = torch.arange(r, device="cuda", dtype=torch.float64)
    if k >= r:
        s = 10.0 ** (-6.25 * i / r)
    else:
        s = torch.where(i < k, 10.0 ** (-4.5 * i / k), 10.0 ** (-7 - 2 * (i - k) / max(1, r - k)))
    return (q1 * s) @ q2.mH


def _cutoff(case):
    return 1e-15 if case["keep"] >= min(case["rows"], case["cols"]) else 1e-11


def _chains(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for k in range(case["chains"]):
        n = int(rng.integers(case["nmin"], case["nmax"] + 1))
        maxdim = int(rng.choice([case["maxdim"] // 2, case["maxdim"]]))
        g = models.chain_graph(n)
        out.append((models.j1j2_chain(n, float(rng.uniform(0.0, 0.5))), _state(g, _sizes(g, lambda e: 8), 1,
                                                                               _gen(seed * 64 + k)), maxdim))
    return out


def prepare(case, seed):
    ctx = _context(case["precision"])
    kind = case["kind"]
    st = dict(case=case, ctx=ctx)
    if kind in ("region", "eigsolve"):
        st.update(_prepare_chain_region(case, seed, ctx))
    elif kind == "environment":
        H, psi, j, L, _ = _chain(dict(case, chi_c=case["chi_r"], chi_r=case["chi_r"]), seed)
        A, W = psi.tensors[j], H.tensors[j]
        a, s, b = Index(A.shape[0]), Index(2), Index(A.shape[2])
        w1, w2 = Index(W.shape[0]), Index(W.shape[3])
        st.update(L=_up(L, [a.prime(), w1, a], ctx), W=_up(W, [w1, s.prime(), s, w2], ctx),
                  A=_up(A, [a, s, b], ctx), out=[b.prime(), w2, b])
    elif kind == "tdvp":
        H, psi, region = _tree_case(case, seed)
        state, sites = from_network(psi, ctx=ctx, dtype=np.complex128)
        (g, Ht), _ = from_network(H, site_index=sites, ctx=ctx, dtype=np.complex128)
        P = ProjTTN(g, Ht).position(state, region)
        P.map_tensors()
        st.update(state=state, H=Ht, envs=P.envs, region=region)
    elif kind == "factorize":
        l, r = Index(case["rows"]), Index(case["cols"])
        st.update(T=_up(_matrix(case, seed), [l, r], ctx), left=[l])
    elif kind == "expand":
        H, psi, j = _expand_case(case, seed)
        state, sites = from_network(psi, ctx=ctx)
        (g, Ht), _ = from_network(H, site_index=sites, ctx=ctx)
        P = ProjTTN(g, Ht)
        P.environment(state, j - 2, j - 1)
        P.environment(state, j + 2, j + 1)
        st.update(state=state, H=Ht, envs=P.envs, region=[j, j + 1], before=[j - 1, j])
    elif kind == "dmrg":
        g = models.chain_graph(case["n"])
        st.update(H=models.heisenberg_chain(case["n"]),
                  psi0=_state(g, _sizes(g, lambda e: case["chi0"]), 1, _gen(seed)))
    else:
        st.update(chains=_chains(case, seed))
    ctx.synchronize()
    return st


# ----------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------


class _Shared:
    """A device tensor of the package as torch sees it (no copy; keeps the storage alive)."""

    def __init__(self, t):
        p = _native.p()
        t.ctx.check(t.ctx.L.nsg_tensor_device_ptr(t.st.h, _native.C.byref(p)))
        size = 16 if t.is_complex() else 8
        strides, s = [], size
        for d in t.shape:
            strides.append(s)
            s *= d
        self.keep = t
        self.__cuda_array_interface__ = dict(shape=t.shape, typestr="<c16" if t.is_complex() else "<f8",
                                             data=(p.value, False), strides=tuple(strides), version=2)


def _torch(t):
    return torch.as_tensor(_Shared(t), device="cuda")


def _problem(cls, st, position):
    P = ProjTTN(st["state"].g, st["H"])
    P.envs = dict(st["envs"])
    P.position(st["state"], position)
    return cls(st["state"], P)


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "region":
        E, left, right, _ = region_step(st["L"], st["W1"], st["W2"], st["R"], st["psi1"], st["psi2"],
                                        direction=case["direction"], krylovdim=3, maxiter=1, cutoff=case["cutoff"],
                                        maxdim=case["maxdim"])
        return dict(energy=np.float64(E), theta=_torch(left * right))
    if kind == "eigsolve":
        lm = LinearMap(_Fixed([st["L"], st["R"], st["W1"], st["W2"]]), st["x"].inds)
        E, x = eigsolve_solver(lm, st["x"], krylovdim=3, maxiter=1)
        return dict(energy=np.float64(E), x=_torch(x))
    if kind == "environment":
        return dict(env=_torch(contract([st["A"], st["L"], st["W"], st["A"].dag().prime()], out=st["out"])))
    if kind == "tdvp":
        u, v = st["region"]
        prob = _problem(ApplyExpProblem, st, st["region"])
        it = RegionIterator(prob, [(st["region"], {})])
        prob = region_iterator_action(prob, it, updater_applyexp,
                                      updater_kwargs=dict(nsites=2, time_step=-1j * case["dt"],
                                                          solver=exponentiate_solver, tol=1e-12),
                                      inserter_kwargs=dict(trunc=dict(cutoff=case["cutoff"], maxdim=case["chi"])))
        return dict(theta=_torch(prob.state[u] * prob.state[v]))
    if kind == "factorize":
        U, C, info = factorize(st["T"], st["left"], cutoff=_cutoff(case), maxdim=min(case["rows"], case["cols"]),
                               spectrum=True)
        return dict(product=_torch(U * C), spectrum=info["spectrum"])
    if kind == "expand":
        u, v = st["region"]
        prob = _problem(EigsolveProblem, st, st["before"])
        it = RegionIterator(prob, [(st["region"], {})])
        prob = region_iterator_action(prob, it, updater_eigsolve,
                                      extracter_kwargs=dict(trunc=dict(cutoff=1e-12, maxdim=case["maxdim"]),
                                                            subspace_algorithm="densitymatrix"),
                                      updater_kwargs=dict(krylovdim=3, maxiter=1),
                                      inserter_kwargs=dict(trunc=dict(cutoff=1e-12, maxdim=case["chi"])))
        return dict(energy=np.float64(prob.eigenvalue), theta=_torch(prob.state[u - 1] * prob.state[u] * prob.state[v]))
    if kind == "dmrg":
        energies = []
        ns.dmrg(st["H"], st["psi0"], nsweeps=case["nsweeps"], nsites=2, ctx=st["ctx"],
                updater_kwargs=dict(krylovdim=3, maxiter=1),
                inserter_kwargs=dict(trunc=dict(cutoff=case["cutoff"], maxdim=case["maxdim"])),
                region_callback=lambda prob, **k: energies.append(prob.eigenvalue))
        return np.array(energies)
    jobs = [batch.dmrg_job(H, psi0, tag=k, nsweeps=case["nsweeps"], maxdim=m, cutoff=1e-10)
            for k, (H, psi0, m) in enumerate(st["chains"])]
    res = batch.SolvePool(workers=case["workers"], precision=case["precision"], tuning={"dc_leaf": 16}).run(jobs)
    if any(r.error for r in res):
        raise RuntimeError([r.error for r in res if r.error][0])
    return np.array([r.value for r in res])


# ----------------------------------------------------------------------------
# work and exact values
# ----------------------------------------------------------------------------


def _heff_flops(a, b, w, d=2):
    return 2.0 * (w * d * d * a * b * (a + b) + w * w * d ** 4 * a * b)


def _fact_flops(m, n, k):
    """Gram product, tridiagonal form, back-transformation and the second factor."""
    r, big = min(m, n), max(m, n)
    return 2.0 * r * r * big + 4.0 / 3.0 * r ** 3 + 4.0 * r * r * k + 2.0 * m * n * k


def _bonds(n, chi):
    return [min(2 ** min(i, n - i), chi) for i in range(n + 1)]


def _sweeps_work(n, chi, w, nsweeps):
    d, f, by = _bonds(n, chi), 0.0, 0.0
    for i in range(1, n):
        f += 3 * _heff_flops(d[i - 1], d[i + 1], w) + _fact_flops(2 * d[i - 1], 2 * d[i + 1], d[i])
        by += 8.0 * (w * d[i - 1] ** 2 + w * d[i + 1] ** 2 + 8 * d[i - 1] * d[i + 1])
    return 2 * nsweeps * f, 2 * nsweeps * by


def work(case):
    kind = case["kind"]
    w = 8 if case.get("model") == "j1j2" else 5
    if kind in ("region", "eigsolve"):
        a, b = case["chi_l"], case["chi_r"]
        f, by = 3 * _heff_flops(a, b, w), 8.0 * (w * (a * a + b * b) + 8 * a * b)
        if kind == "region":
            c = case["chi_c"]
            k = min(2 * a, 2 * b, case["maxdim"])
            f += 8.0 * a * b * c + _fact_flops(2 * a, 2 * b, k) + 8.0 * a * b * k
            by += 8.0 * (2 * a * c + 2 * b * c)
        return dict(bytes=by, flops=f)
    if kind == "environment":
        a, b = case["chi_l"], case["chi_r"]
        return dict(bytes=8.0 * (w * a * a + w * b * b + 2 * a * b),
                    flops=2.0 * (2 * w * a * a * b + 4 * w * w * a * b + 2 * w * a * b * b))
    if kind == "tdvp":
        c = case["chi"]
        if case["graph"] == "tree":
            size, envs, f = 4.0 * c ** 3, 3, 8.0 * 6 * 4 * 3 * 3 * c ** 4
            rows, cols = 2 * c * c, 2 * c
        else:
            size, envs, f = 4.0 * c ** 2, 2, 8.0 * 6 * 3 * 4 * 2 * c ** 3
            rows, cols = 2 * c, 2 * c
        return dict(bytes=16.0 * (2 * size + envs * 3 * c * c), flops=f + 4 * _fact_flops(rows, cols, c))
    if kind == "factorize":
        m, n, z = case["rows"], case["cols"], 4.0 if case["complex"] else 1.0
        return dict(bytes=(16.0 if case["complex"] else 8.0) * 2 * m * n,
                    flops=z * (_fact_flops(m, n, case["keep"]) + 2.0 * m * n * case["keep"]))
    if kind == "expand":
        c = case["chi"]
        e = min(2 * c, case["maxdim"])
        f = 3 * _heff_flops(e, c, 5) + _fact_flops(2 * e, 2 * c, c) + _fact_flops(2 * c, 5 * c, e - c)
        return dict(bytes=8.0 * (2 * 5 * c * c + 3 * 2 * c * c + 8 * c * c), flops=f + 2.0 * 2 * 2 * c * e * 2 * c)
    if kind == "dmrg":
        f, by = _sweeps_work(case["n"], case["maxdim"], 5, case["nsweeps"])
        return dict(bytes=by, flops=f)
    f, by = _sweeps_work((case["nmin"] + case["nmax"]) // 2, 3 * case["maxdim"] // 4, 8, case["nsweeps"])
    return dict(bytes=case["chains"] * by, flops=case["chains"] * f)


def _apply(fixed, x, lx):
    T, lt = x, lx
    for t, l in fixed:
        T, lt = _dot(T, lt, t, l)
    return T.permute([lt.index(n) for n in _bra(lx)])


def _lowest(alpha, beta):
    """Lowest eigenpair of the tridiagonal, by cyclic Jacobi rotations (which fix its sign)."""
    k = len(alpha)
    A = np.diag(alpha) + np.diag(beta[: k - 1], 1) + np.diag(beta[: k - 1], -1)
    V = np.eye(k)
    for _ in range(60):
        for p in range(k - 1):
            for q in range(p + 1, k):
                if abs(A[p, q]) < 1e-300:
                    continue
                th = (A[q, q] - A[p, p]) / (2 * A[p, q])
                t = (1.0 if th >= 0 else -1.0) / (abs(th) + math.sqrt(th * th + 1))
                c = 1 / math.sqrt(t * t + 1)
                J = np.eye(k)
                J[p, p] = J[q, q] = c
                J[p, q], J[q, p] = t * c, -t * c
                A, V = J.T @ A @ J, V @ J
    i = int(np.argmin(np.diag(A)))
    return float(A[i, i]), V[:, i]


def _lanczos(fixed, x, lx, steps=3):
    V, alpha, beta = [x / x.norm()], [], []
    for j in range(steps):
        w = _apply(fixed, V[j], lx)
        a = 0.0
        for _ in range(2):
            for i, v in enumerate(V):
                c = torch.sum(v * w)
                w = w - c * v
                if i == j:
                    a += float(c)
        alpha.append(a)
        beta.append(float(w.norm()))
        if j + 1 < steps:
            V.append(w / w.norm())
    E, y = _lowest(alpha, beta)
    z = sum(float(c) * v for c, v in zip(y, V))
    return E, z / z.norm()


def _kept(p, cutoff, maxdim):
    """Number of descending weights p that the truncation keeps."""
    n = min(len(p), maxdim) if maxdim else len(p)
    total, err = float(p.sum()), float(p[n:].sum())
    while n > 1 and err + float(p[n - 1]) < cutoff * total:
        err += float(p[n - 1])
        n -= 1
    return n


def _cut(mat, cutoff, maxdim):
    """mat with its singular values truncated, and the kept ones' squares."""
    U, S, Vh = torch.linalg.svd(mat, full_matrices=False)
    k = _kept((S * S).cpu().numpy(), cutoff, maxdim)
    return (U[:, :k] * S[:k]) @ Vh[:k], (S[:k] * S[:k]).cpu().numpy()


def _two_site(psi, u, v, dtype):
    return _dot(*_site(psi, u, dtype), *_site(psi, v, dtype))


def _fixed(H, psi, region, dtype):
    out = []
    for v in region:
        for w in psi.graph.neighbors(v):
            if w not in region:
                e = psi.graph.edge_key(w, v)
                out.append((_env(H, psi, w, v, dtype), [("b", e), ("w", e), ("l", e)]))
    return out + [_site(H, v, dtype) for v in region]


def exact(case, seed):
    kind = case["kind"]
    f64 = torch.float64
    if kind in ("region", "eigsolve"):
        H, psi, j, _, _ = _chain(case, seed)
        x, lx = _two_site(psi, j, j + 1, f64)
        E, y = _lanczos(_fixed(H, psi, [j, j + 1], f64), x, lx)
        if kind == "eigsolve":
            return dict(energy=np.float64(E), x=y)
        a, s, t, b = y.shape
        theta, _ = _cut(y.reshape(a * s, t * b), case["cutoff"], case["maxdim"])
        return dict(energy=np.float64(E), theta=theta.reshape(a, s, t, b))
    if kind == "environment":
        H, psi, j, _, _ = _chain(dict(case, chi_c=case["chi_r"], chi_r=case["chi_r"]), seed)
        return dict(env=_env(H, psi, j, j + 1, f64))
    if kind == "tdvp":
        c128 = torch.complex128
        H, psi, (u, v) = _tree_case(case, seed)
        x, lx = _two_site(psi, u, v, c128)
        fixed, term, y = _fixed(H, psi, [u, v], c128), x, x
        for n in range(1, 400):
            term = _apply(fixed, term, lx) * (-1j * case["dt"] / n)
            y = y + term
            if float(term.norm()) < 1e-18:
                break
        rows = math.prod(y.shape[: len(_site(psi, u, c128)[1]) - 1])
        theta, _ = _cut(y.reshape(rows, -1), case["cutoff"], case["chi"])
        return dict(theta=theta.reshape(y.shape))
    if kind == "factorize":
        product, p = _cut(_matrix(case, seed), _cutoff(case), min(case["rows"], case["cols"]))
        return dict(product=product, spectrum=p)
    if kind == "expand":
        H, psi, j = _expand_case(case, seed)
        A, la = _site(psi, j - 1, f64)
        eL, ea = psi.graph.edge_key(j - 2, j - 1), ("l", psi.graph.edge_key(j - 1, j))
        ew = ("w", ea[1])
        ket = [x for x in la if x != ea]
        T, lt = _dot(A, la, _env(H, psi, j - 2, j - 1, f64), [("b", eL), ("w", eL), ("l", eL)])
        T, lt = _dot(T, lt, *_site(H, j - 1, f64))
        X = T.permute([lt.index(n) for n in _bra(ket) + [ew, ea]])
        X = X.reshape(X.shape[0] * X.shape[1], -1)
        Am = A.permute([la.index(n) for n in ket + [ea]]).reshape(X.shape[0], -1)
        chi, rows = Am.shape[1], Am.shape[0]
        grow = max(0, min(math.ceil(1.5 * chi), rows - chi, case["maxdim"] - chi))
        X = X - Am @ (Am.T @ X)
        p, U = torch.linalg.eigh(X @ X.T)
        p, U = p.flip(0).clamp(min=0), U.flip(1)
        U = U[:, : _kept(p.cpu().numpy(), 1e-12, grow)]
        U = U - Am @ (Am.T @ U)
        Q = torch.cat([Am, U], 1)
        x, lx = _two_site(psi, j, j + 1, f64)
        lift = torch.cat([torch.eye(chi, dtype=f64, device="cuda"), U.T @ Am], 0)
        x = torch.tensordot(lift, x, dims=([1], [0]))
        env, le = _env(H, psi, j - 2, j - 1, f64), [("b", eL), ("w", eL), ("l", eL)]
        e, l = _dot(Q.reshape([A.shape[la.index(n)] for n in ket] + [-1]), ket + [ea], env, le)
        e, l = _dot(e, l, *_site(H, j - 1, f64))
        e, l = _dot(e, l, Q.reshape([A.shape[la.index(n)] for n in ket] + [-1]), _bra(ket) + [("b", ea[1])])
        fixed = [f for f in _fixed(H, psi, [j, j + 1], f64) if ("l", ea[1]) not in f[1]]
        E, y = _lanczos([(e, l)] + fixed, x, lx)
        shape = y.shape
        theta, _ = _cut(y.reshape(shape[0] * shape[1], -1), 1e-12, case["chi"])
        theta = (Q @ theta.reshape(shape[0], -1)).reshape([A.shape[la.index(n)] for n in ket] + list(shape[1:]))
        return dict(energy=np.float64(E), theta=theta)
    return None
