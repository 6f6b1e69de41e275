"""The divide and conquer through `eigen_hermitian` at the orders where its forms change
(leaf only, one cluster, a launch per step, tensor-core merges), on spectra that deflate
little, much, and in exact multiplets, against numpy.  A backward-stable symmetric
eigensolver leaves residuals and orthogonality at a modest multiple of n eps of the norm;
the bounds are 20 n eps (measured errors sit well below n eps)."""
import numpy as np
import pytest

from networksolvers_gb300.itensors import DTensor, Index, eigen_hermitian, factorize

pytestmark = pytest.mark.gpu
EPS = 2.3e-16


def check(ctx, A, leaf=0):
    n = A.shape[0]
    i = Index(n)
    ctx.set_tuning("dc_leaf", leaf)
    try:
        ev, U, _ = eigen_hermitian(DTensor.from_numpy(A, [i.prime(), i]), [i], cutoff=0.0, maxdim=n)
        U = U.to_numpy()
    finally:
        ctx.set_tuning("dc_leaf", 0)
    norm = max(np.linalg.norm(A, 2), 1e-300)
    bound = 20 * n * EPS
    k = U.shape[1]
    assert np.linalg.norm(U.conj().T @ U - np.eye(k), 2) < bound
    # rho [bra, ket] = A has the eigenvectors A U = U diag(ev)
    assert np.linalg.norm(A @ U - U * ev, 2) < bound * norm
    ref = np.linalg.eigvalsh(A)[::-1][:k]
    assert np.max(np.abs(ev - ref)) < bound * norm


def spectra(rng, n, kind):
    if kind == "random":
        return rng.standard_normal(n)
    if kind == "graded":
        return 10.0 ** (-16.0 * np.arange(n) / n)
    if kind == "multiplets":
        return np.repeat(rng.standard_normal((n + 4) // 5), 5)[:n]
    if kind == "clustered":
        return np.where(np.arange(n) % 2 == 0, 1.0, 1.0 + 1e-15 * np.arange(n)) + 1e-9 * (np.arange(n) % 7 == 0)
    return np.concatenate([np.ones(n - n // 3), np.zeros(n // 3)])


@pytest.mark.parametrize("kind", ["random", "graded", "multiplets", "clustered", "projector"])
@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 16, 17, 31, 33, 64, 65, 129, 160, 161, 230, 513])
def test_orders_and_spectra(nsg_ctx, n, kind):
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = (Q * spectra(rng, n, kind)) @ Q.T
    check(nsg_ctx, 0.5 * (A + A.T))


@pytest.mark.parametrize("leaf", [4, 5, 13, 32])
@pytest.mark.parametrize("n", [5, 33, 100, 200])
def test_leaf_orders(nsg_ctx, n, leaf):
    rng = np.random.default_rng(n + leaf)
    A = rng.standard_normal((n, n))
    check(nsg_ctx, A + A.T, leaf)


@pytest.mark.parametrize("n", [2, 9, 50, 170])
def test_complex(nsg_ctx, n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    check(nsg_ctx, A + A.conj().T)


@pytest.mark.parametrize("scale", [1e-140, 1e140])
@pytest.mark.parametrize("n", [6, 40, 200])
def test_extreme_scales(nsg_ctx, n, scale):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    check(nsg_ctx, scale * (A + A.T))


@pytest.mark.parametrize("n", [1, 8, 40, 200])
def test_diagonal_and_zero(nsg_ctx, n):
    check(nsg_ctx, np.diag(np.arange(n, 0, -1.0)))
    check(nsg_ctx, np.zeros((n, n)))


@pytest.mark.parametrize("n", [50, 140, 300, 500])
def test_rank_one_falls_by_eps_per_row(nsg_ctx, n):
    """The reduction of a matrix of ones leaves tridiagonal blocks down to the end of the
    exponent range."""
    check(nsg_ctx, np.ones((n, n)))
    v = np.cos(np.arange(n))
    check(nsg_ctx, np.outer(v, v) * 1e-60)


@pytest.mark.parametrize("precision", ["ozaki", "ozaki8"])
@pytest.mark.parametrize("n", [257, 400, 530, 700])
def test_tensor_core_merges(nsg_ctx, n, precision):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    nsg_ctx.set_precision(precision)
    try:
        check(nsg_ctx, A + A.T)
    finally:
        nsg_ctx.set_precision("fp64")


def test_equal_eigenvalues_up_to_rounding(nsg_ctx):
    """Gram matrices of orthogonal matrices and projectors: leaves of equal diagonal entries and
    off-diagonal ones at the rounding level."""
    rng = np.random.default_rng(0)
    for rep in range(60):
        n = (24, 64, 100, 200)[rep % 4]
        Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
        for A in (Q, Q[:, : n // 2] @ Q[:, : n // 2].T, np.eye(n) + 1e-16 * rng.standard_normal((n, n))):
            i, j = Index(n), Index(n)
            U, C, _ = factorize(DTensor.from_numpy(A, [i, j]), [i], cutoff=0.0, maxdim=n)
            U, C = U.to_numpy(), C.to_numpy()
            assert np.linalg.norm(U @ C - A, 2) < 20 * n * 2.3e-16
            assert np.linalg.norm(U.T @ U - np.eye(n), 2) < 20 * n * 2.3e-16
