"""The split products' slicing at the edges of its tiles: rows and depths around multiples of
32, depths beyond one shared-memory slab, rows of very different scale, and entries at the
ends of the exponent range.  Bound: six slices hold each operand to 2^-43 of its row's (or
column's) scale, so a product of depth K is within 4 K 2^-42 of the product of the scales;
eight hold 2^-57, and the pair of FP32 accumulators (2^-48 of partial sums of at most K of
the scales' product) bounds: 4 K 2^-48."""
import numpy as np
import pytest

from networksolvers_gb300.itensors import DTensor, Index, contract

pytestmark = pytest.mark.gpu


def rnd(rng, shape, cplx):
    x = rng.standard_normal(shape)
    return x + 1j * rng.standard_normal(shape) if cplx else x


@pytest.mark.parametrize("precision,bits", [("ozaki", 42), ("ozaki8", 48)])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n,k", [(64, 32, 64), (65, 33, 97), (96, 64, 416), (130, 70, 417), (64, 40, 1000),
                                   (300, 200, 3329), (70, 64, 7000), (1024, 700, 130)])
def test_slices_every_orientation(nsg_ctx, precision, bits, cplx, m, n, k):
    rng = np.random.default_rng(m + n + k)
    a = rnd(rng, (m, k), cplx) * 10.0 ** rng.integers(-9, 9, (m, 1))
    b = rnd(rng, (k, n), cplx) * 10.0 ** rng.integers(-9, 9, (1, n))
    a[:, rng.integers(0, k)] *= 1e-7
    ref = a @ b
    bound = (8 if cplx else 4) * k * 2.0 ** -bits * np.abs(a).max(1)[:, None] * np.abs(b).max(0)[None]
    i, j, l = Index(m), Index(n), Index(k)
    nsg_ctx.set_precision(precision)
    try:
        for ta in (False, True):
            A = DTensor.from_numpy(a.T, [l, i]) if ta else DTensor.from_numpy(a, [i, l])
            for tb in (False, True):
                B = DTensor.from_numpy(b.T, [j, l]) if tb else DTensor.from_numpy(b, [l, j])
                got = contract([A, B], out=[i, j]).to_numpy()
                assert np.all(np.abs(got - ref) <= bound + 1e-14 * np.abs(ref)), (ta, tb)
    finally:
        nsg_ctx.set_precision("fp64")


@pytest.mark.parametrize("precision,bits", [("ozaki", 42), ("ozaki8", 48)])
@pytest.mark.parametrize("k", [384, 385, 416, 777])
def test_chunks_of_one_pass_over_k(nsg_ctx, precision, bits, k):
    """Depths around the exact chunk's length where K is not split over CTAs (100 output
    tiles), with every entry's digits near their largest value and of one sign."""
    rng = np.random.default_rng(k)
    m, n = 1270, 630
    a, b = 1.0 - 2.0 ** -40 * rng.random((m, k)), 1.0 - 2.0 ** -9 * (1 + rng.random((k, n)))
    i, j, l = Index(m), Index(n), Index(k)
    nsg_ctx.set_precision(precision)
    try:
        got = contract([DTensor.from_numpy(a, [i, l]), DTensor.from_numpy(b, [l, j])], out=[i, j]).to_numpy()
    finally:
        nsg_ctx.set_precision("fp64")
    assert np.max(np.abs(got - a @ b)) <= 4 * k * 2.0 ** -bits


@pytest.mark.parametrize("precision", ["ozaki", "ozaki8"])
def test_slices_batched(nsg_ctx, precision):
    rng = np.random.default_rng(4)
    m, n, k, q = 70, 40, 65, 9
    a, b = rng.standard_normal((m, k, q)), rng.standard_normal((k, n))
    i, j, l, x = Index(m), Index(n), Index(k), Index(q)
    nsg_ctx.set_precision(precision)
    try:
        got = contract([DTensor.from_numpy(a, [i, l, x]), DTensor.from_numpy(b, [l, j])], out=[i, j, x]).to_numpy()
    finally:
        nsg_ctx.set_precision("fp64")
    ref = np.einsum("ilx,lj->ijx", a, b)
    assert np.max(np.abs(got - ref)) < 4 * k * 2.0 ** -42 * np.abs(a).max() * np.abs(b).max()


@pytest.mark.parametrize("precision", ["ozaki", "ozaki8"])
def test_zero_extreme_and_non_finite_rows(nsg_ctx, precision):
    rng = np.random.default_rng(5)
    m, n, k = 128, 64, 128
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    a[0] = 0.0
    a[1] *= 1e-300
    a[2] *= 1e290
    a[3, 5:] = 0.0
    a[4, ::2] = 0.5
    i, j, l = Index(m), Index(n), Index(k)
    nsg_ctx.set_precision(precision)
    try:
        got = contract([DTensor.from_numpy(a, [i, l]), DTensor.from_numpy(b, [l, j])], out=[i, j]).to_numpy()
        bound = 4 * k * 2.0 ** -42 * np.abs(a).max(1)[:, None] * np.abs(b).max(0)[None]
        assert np.all(np.abs(got - a @ b) <= bound + 1e-14 * np.abs(a @ b))
        assert np.all(got[0] == 0.0)
        for bad in (np.inf, np.nan):
            a2 = a.copy()
            a2[7, 3] = bad
            got2 = contract([DTensor.from_numpy(a2, [i, l]), DTensor.from_numpy(b, [l, j])], out=[i, j]).to_numpy()
            assert not np.any(np.isfinite(got2[7]))
            keep = np.arange(m) != 7
            assert np.array_equal(got2[keep], got[keep])
    finally:
        nsg_ctx.set_precision("fp64")


def test_partial_products_of_one_term_at_a_time(nsg_ctx):
    """A complex product whose K is split keeps the partial products of its four terms; where the
    budget has no room for them, of one term at a time, with the same result."""
    from networksolvers_gb300 import _native
    rng = np.random.default_rng(3)
    m, n, k = 512, 128, 1280
    a, b = rnd(rng, (m, k), True), rnd(rng, (k, n), True)
    i, j, l = Index(m), Index(n), Index(k)
    got, budget = [], 0
    try:
        for _ in range(2):
            ctx = _native.Context(0, hbm_budget=budget, precision="ozaki")
            _native.set_default_context(ctx)
            A, B = DTensor.from_numpy(a, [i, l]), DTensor.from_numpy(b, [l, j])
            C = contract([A, B], out=[i, j])
            got.append(C.to_numpy())
            budget = ctx.memory()[1] - 2 * 8 * 2 * m * n  # two terms' partial products, of two splits or more
            del A, B, C
    finally:
        _native.set_default_context(nsg_ctx)
    assert np.array_equal(got[0], got[1])
    assert np.max(np.abs(got[0] - a @ b)) < 8 * k * 2.0 ** -42 * np.abs(a).max() * np.abs(b).max()


@pytest.mark.parametrize("p,q", [(4096, 16), (4097, 16), (4096, 2049)])
def test_depth_beyond_a_grid(nsg_ctx, p, q):
    """Slices of 512 slabs of the depth and one more, and of more than a grid has rows (65535 of
    128), of operands that repeat."""
    rng = np.random.default_rng(8)
    m, n = 64, 32
    a, b = rng.standard_normal((m, p)), rng.standard_normal((p, n))
    i, j, l = Index(m), Index(n), Index(p * q)
    nsg_ctx.set_precision("ozaki")
    try:
        A, B = DTensor.from_numpy(np.tile(a.T, (q, 1)).T, [i, l]), DTensor.from_numpy(np.tile(b.T, (1, q)).T, [l, j])
        got = contract([A, B], out=[i, j]).to_numpy()
        del A, B
    finally:
        nsg_ctx.set_precision("fp64")
    bound = 4 * p * q * 2.0 ** -42 * np.abs(a).max(1)[:, None] * np.abs(b).max(0)[None]
    assert np.all(np.abs(got - q * (a @ b)) <= bound)


@pytest.mark.parametrize("cplx", [False, True])
def test_eight_slices_batched_and_at_the_ends_of_the_range(nsg_ctx, cplx):
    """The batched slicing and rows of extreme scale to the eight-slice bound: one slice less would
    be 2^6 above it."""
    rng = np.random.default_rng(6)
    m, n, k, q = 128, 64, 129, 5
    a, b = rnd(rng, (m, k, q), cplx), rnd(rng, (k, n), cplx)
    a[0] = 0.0
    a[1] *= 1e-300
    a[2] *= 1e290
    a[3, 5:] = 0.0
    a[4, ::2] = 0.5
    i, j, l, x = Index(m), Index(n), Index(k), Index(q)
    nsg_ctx.set_precision("ozaki8")
    try:
        got = contract([DTensor.from_numpy(a, [i, l, x]), DTensor.from_numpy(b, [l, j])], out=[i, j, x]).to_numpy()
    finally:
        nsg_ctx.set_precision("fp64")
    ref = np.einsum("ilx,lj->ijx", a, b)
    scales = np.abs(a).max(1)[:, None, :] * np.abs(b).max(0)[None, :, None]
    bound = (8 if cplx else 4) * k * 2.0 ** -48 * scales
    assert np.all(np.abs(got - ref) <= bound + 1e-14 * np.abs(ref))
    assert np.all(got[0] == 0.0)
