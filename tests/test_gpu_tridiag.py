"""The resident tridiagonalisation, over one cluster and over all SMs, through
`eigen_hermitian`: orders around its row blocks (128) and the number of SMs (one column per
CTA and more), the largest orders that fit shared memory and the first that do not, and
matrices whose columns need no reflection, span the exponent range or are not finite.  A
backward-stable symmetric eigensolver leaves residuals and orthogonality at a modest multiple
of n eps of the norm; the bounds are 20 n eps."""
import numpy as np
import pytest

from networksolvers_gb300._native import NsgError
from networksolvers_gb300.itensors import DTensor, Index, eigen_hermitian

pytestmark = pytest.mark.gpu
EPS = 2.3e-16


def check(ctx, A, path, vectors=True):
    n = A.shape[0]
    i = Index(n)
    ctx.set_tuning("tridiag", path)
    try:
        ev, U, _ = eigen_hermitian(DTensor.from_numpy(A, [i.prime(), i]), [i], cutoff=0.0, maxdim=n if vectors else 2)
        U = U.to_numpy()
    finally:
        ctx.set_tuning("tridiag", 0)
    norm = np.linalg.norm(A, 2) if vectors else np.linalg.norm(A)
    bound = 20 * n * EPS
    k = U.shape[1]
    assert np.linalg.norm(U.conj().T @ U - np.eye(k), 2) < bound
    assert np.linalg.norm(A @ U - U * ev, 2) <= bound * norm
    if vectors:
        assert np.max(np.abs(ev - np.linalg.eigvalsh(A)[::-1][:k])) <= bound * norm


def hermitian(rng, n, cplx):
    A = rng.standard_normal((n, n))
    if cplx:
        A = A + 1j * rng.standard_normal((n, n))
    return A + A.conj().T


@pytest.mark.parametrize("path", [2, 8, 16, -1])
@pytest.mark.parametrize("cplx", [False, True])
def test_orders(nsg_ctx, path, cplx):
    rng = np.random.default_rng(path + 20)
    for n in (3, 4, 5, 16, 17, 33, 127, 128, 129, 151, 152, 153, 257, 305):
        check(nsg_ctx, hermitian(rng, n, cplx), path)


@pytest.mark.parametrize("path", [4, -1])
@pytest.mark.parametrize("cplx", [False, True])
def test_special_matrices(nsg_ctx, path, cplx):
    rng = np.random.default_rng(7)
    n = 140
    full = hermitian(rng, n, cplx)
    blocks = full.copy()
    blocks[:60, 60:] = blocks[60:, :60] = 0.0
    s = 10.0 ** (-14.0 * rng.permutation(n) / n)
    cases = [np.diag(rng.standard_normal(n)).astype(full.dtype), np.triu(np.tril(full, 1), -1), blocks,
             full * s[:, None] * s[None, :], full * 1e-140, full * 1e140, np.ones((n, n), full.dtype)]
    decoupled = full.copy()  # couplings far below the rounding of the rest
    decoupled[0, 1:] *= 1e-170
    decoupled[1:, 0] *= 1e-170
    for A in cases + [decoupled]:
        check(nsg_ctx, A, path)


@pytest.mark.parametrize("n,cplx", [(1774, False), (1775, False), (1210, True), (1211, True)])
def test_largest_resident_orders(nsg_ctx, n, cplx):
    check(nsg_ctx, hermitian(np.random.default_rng(n), n, cplx), -1, vectors=False)


@pytest.mark.parametrize("path", [8, -1])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite(nsg_ctx, path, bad):
    A = hermitian(np.random.default_rng(1), 200, False)
    A[70, 20] = A[20, 70] = bad
    with pytest.raises(NsgError):
        check(nsg_ctx, A, path, vectors=False)
    check(nsg_ctx, hermitian(np.random.default_rng(2), 200, False), path)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n", [40, 140])
def test_norms_whose_squares_leave_the_range(nsg_ctx, n, cplx):
    full = hermitian(np.random.default_rng(n), n, cplx)
    for path in (4, -1):
        for s in (1e-155, 1e-160, 1e-200, 1e-280, 1e160, 1e280):
            check(nsg_ctx, full * s, path)
