"""Contraction orders and layouts: random networks whose tensors hold their labels in
random orders, with conjugated operands and requested result orders, and linear maps with
fixed-only parts, against numpy's einsum.  Tolerance: the summed depth (at most a few
thousand products in any order) times eps of the absolute result."""
import itertools
import string

import numpy as np
import pytest

from networksolvers_gb300 import _native
from networksolvers_gb300.itensors import DTensor, Index, contract
from networksolvers_gb300.network import LinearMap

pytestmark = pytest.mark.gpu


def rnd(rng, shape, cplx):
    x = rng.standard_normal(shape)
    return x + 1j * rng.standard_normal(shape) if cplx else x


def network(rng, n, cplx):
    """n tensors: a random spanning tree of shared labels plus a few extra ones, at most one
    open label each (so the result has at most 4^6 entries), in shuffled orders."""
    pairs = [(int(rng.integers(0, k)), k) for k in range(1, n)]
    for _ in range(int(rng.integers(0, n))):
        a, b = rng.choice(n, 2, replace=False)
        pairs.append((int(min(a, b)), int(max(a, b))))
    labels = [[] for _ in range(n)]
    inds, opened = [], []
    for a, b in pairs:
        i = Index(int(rng.integers(1, 6)))
        inds.append(i)
        labels[a].append(i)
        labels[b].append(i)
    for k in range(n):
        if rng.integers(0, 3) > 0:
            i = Index(int(rng.integers(1, 5)))
            inds.append(i)
            opened.append(i)
            labels[k].append(i)
    for l in labels:
        rng.shuffle(l)
    rng.shuffle(opened)
    arrays = [rnd(rng, [i.dim for i in l], cplx) for l in labels]
    return labels, arrays, opened


def einsum(labels, arrays, out):
    letters = {}
    for l in labels:
        for i in l:
            letters.setdefault(i, string.ascii_letters[len(letters)])
    spec = ",".join("".join(letters[i] for i in l) for l in labels) + "->" + "".join(letters[i] for i in out)
    return np.einsum(spec, *arrays, optimize="optimal")


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("seed,n", list(itertools.product(range(6), [2, 3, 4, 5, 6])))
def test_random_networks(nsg_ctx, seed, n, cplx):
    rng = np.random.default_rng(100 * seed + n)
    labels, arrays, out = network(rng, n, cplx)
    conj = [cplx and bool(rng.integers(0, 2)) for _ in range(n)]
    ts = [DTensor.from_numpy(a, l) for a, l in zip(arrays, labels)]
    got = contract([t.dag() if c else t for t, c in zip(ts, conj)], out=out).to_numpy()
    ref = einsum(labels, [a.conj() if c else a for a, c in zip(arrays, conj)], out)
    mag = einsum(labels, [np.abs(a) for a in arrays], out)
    assert got.shape == ref.shape
    assert np.all(np.abs(got - ref) <= 1e-12 * mag + 1e-300)


class _Map:
    def __init__(self, tensors):
        self.tensors = tensors

    def map_tensors(self):
        return self.tensors


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("seed", range(8))
def test_linear_map_layouts(nsg_ctx, seed, cplx):
    """A two-site effective Hamiltonian with every tensor's labels in a random order, applied
    twice (the second application uses the fixed-only parts kept by the first)."""
    rng = np.random.default_rng(seed)
    a, b = (Index(int(rng.integers(1, 12))) for _ in range(2))
    s1, s2 = (Index(int(rng.integers(1, 4))) for _ in range(2))
    w1, w2, w3 = (Index(int(rng.integers(1, 5))) for _ in range(3))
    legs = [[a.prime(), w1, a], [b.prime(), w3, b], [w1, s1.prime(), s1, w2], [w2, s2.prime(), s2, w3]]
    x = [a, s1, s2, b]
    for l in legs + [x]:
        rng.shuffle(l)
    arrays = [rnd(rng, [i.dim for i in l], cplx) for l in legs]
    lm = LinearMap(_Map([DTensor.from_numpy(t, l) for t, l in zip(arrays, legs)]), x)
    for _ in range(2):
        v = rnd(rng, [i.dim for i in x], cplx)
        got = lm(DTensor.from_numpy(v, x)).to_numpy()
        out = [i.prime() for i in x]
        ref = einsum(legs + [x], arrays + [v], out)
        mag = einsum(legs + [x], [np.abs(t) for t in arrays] + [np.abs(v)], out)
        assert np.all(np.abs(got - ref) <= 1e-12 * mag + 1e-300)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("ozaki", 1e-10)])
@pytest.mark.parametrize("d,k,b", [(2, 64, 32), (2, 80, 40), (31, 64, 3), (32, 64, 5), (2, 63, 40), (2, 80, 31)])
def test_thin_batched_products(nsg_ctx, precision, tol, d, k, b):
    """The contracted label between a small free label and a large one, on either side (a batched
    product d columns wide, or one wide product of the permuted operand), at the edges of the rule."""
    rng = np.random.default_rng(d + k + b)
    m = 96
    p, q, s, r = Index(m), Index(k), Index(d), Index(b)
    x, y = rng.standard_normal((m, k)), rng.standard_normal((d, k, b))
    nsg_ctx.set_precision(precision)
    try:
        X, Y = DTensor.from_numpy(x, [p, q]), DTensor.from_numpy(y, [s, q, r])
        got = contract([X, Y], out=[p, s, r]).to_numpy()
        swapped = contract([Y, X], out=[s, r, p]).to_numpy()
    finally:
        nsg_ctx.set_precision("fp64")
    ref = np.einsum("pq,sqr->psr", x, y)
    bound = tol * np.abs(x).max() * np.abs(y).max() * k
    assert np.max(np.abs(got - ref)) < bound
    assert np.max(np.abs(swapped - ref.transpose(1, 2, 0))) < bound


@pytest.mark.parametrize("precision", ["fp64", "ozaki"])
def test_thin_batches_without_room_for_a_copy(nsg_ctx, precision):
    """A product batched over thin slices whose operand's permuted copy (and slices) the budget
    does not hold runs as it is, with the same result, and nothing is left behind."""
    rng = np.random.default_rng(11)
    s, k, b, n = 2, 512, 640, 256
    x, y = rng.standard_normal((s, k, b)), rng.standard_normal((k, n))
    i, j, l, q = Index(s), Index(n), Index(k), Index(b)
    out_bytes = 8 * s * n * b
    try:
        ctx = _native.Context(0, hbm_budget=x.nbytes + y.nbytes + out_bytes + (1 << 16), precision=precision)
        _native.set_default_context(ctx)
        A, B = DTensor.from_numpy(x, [i, l, q]), DTensor.from_numpy(y, [l, j])
        before = ctx.memory()[0]
        ref = np.einsum("slb,ln->snb", x, y)
        for out, axes in (([i, j, q], (0, 1, 2)), ([j, i, q], (1, 0, 2))):
            C = contract([A, B], out=out)
            got = C.to_numpy().transpose(axes)
            assert np.linalg.norm(got - ref) <= 1e-13 * np.linalg.norm(ref)
            del C
            assert ctx.memory()[0] == before
        del A, B
    finally:
        _native.set_default_context(nsg_ctx)
