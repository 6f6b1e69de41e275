"""The one-launch Lanczos step through `eigsolve_solver` against the oracle: every number of
vectors it holds in registers, the grouped form, and more than it takes (separate launches); one
CTA, a CTA's share plus or minus a few elements, one and two CTAs per SM.  Both sides are the
same Krylov space by a stable recurrence; up to six vectors the bound is 1e-12, beyond that
1e-10, for the recurrence's amplification of rounding."""
import numpy as np
import pytest

from networksolvers_gb300._native import NsgError
from networksolvers_gb300.itensors import DTensor
from networksolvers_gb300.sweep import eigsolve_solver, exponentiate_solver
from oracle import krylov as ok
from test_gpu_kernels import _chain_heff, _device_map

pytestmark = pytest.mark.gpu


def heff(L, W1, W2, R):
    def f(x):
        y = np.tensordot(L, x, (2, 0))                      # p w s x b
        y = np.einsum("pwsxb,wtsv->ptvxb", y, W1, optimize=True)
        y = np.einsum("ptvxb,vuxz->ptuzb", y, W2, optimize=True)
        return np.einsum("ptuzb,qzb->ptuq", y, R, optimize=True)
    return f


def run(ctx, chi_l, chi_r, krylovdim, cplx, tol):
    rng = np.random.default_rng(chi_l + chi_r + krylovdim)
    L, W1, W2, R = _chain_heff(rng, chi_l, chi_r, cplx=cplx)
    lm, inds = _device_map(L, W1, W2, R)
    x0 = rng.standard_normal((chi_l, 2, 2, chi_r)) + (1j * rng.standard_normal((chi_l, 2, 2, chi_r)) if cplx else 0)
    lam, x = eigsolve_solver(lm, DTensor.from_numpy(x0, inds), krylovdim=krylovdim, maxiter=1)
    lam_o, x_o = ok.eigsolve_lanczos(heff(L, W1, W2, R), x0, krylovdim=krylovdim, maxiter=1)
    x = x.to_numpy()
    assert abs(lam - lam_o) <= tol * abs(lam_o)
    assert abs(abs(np.vdot(x, x_o)) - 1) < tol
    assert abs(np.linalg.norm(x) - 1) < 1e-13


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("krylovdim", [1, 2, 3, 4, 5, 6, 9, 16, 17, 19])
def test_numbers_of_vectors(nsg_ctx, krylovdim, cplx):
    run(nsg_ctx, 20, 37, krylovdim, cplx, 1e-12 if krylovdim <= 6 else 1e-10)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("chi_l,chi_r", [(1, 2), (1, 128), (3, 43), (16, 16), (61, 67), (140, 139), (250, 301)])
def test_lengths(nsg_ctx, chi_l, chi_r, cplx):
    run(nsg_ctx, chi_l, chi_r, 3, cplx, 1e-12)


def test_two_ctas_per_sm(nsg_ctx):
    run(nsg_ctx, 725, 724, 3, False, 1e-12)


@pytest.mark.parametrize("bad", [0.0, np.nan])
def test_zero_and_non_finite_vectors(nsg_ctx, bad):
    rng = np.random.default_rng(0)
    lm, inds = _device_map(*_chain_heff(rng, 30, 30))
    with pytest.raises(NsgError):
        eigsolve_solver(lm, DTensor.from_numpy(np.full((30, 2, 2, 30), bad), inds), krylovdim=3, maxiter=1)


@pytest.mark.parametrize("scale", [1e-150, 1e150])
def test_extreme_norms(nsg_ctx, scale):
    rng = np.random.default_rng(5)
    H = _chain_heff(rng, 12, 10)
    lm, inds = _device_map(*H)
    x0 = rng.standard_normal((12, 2, 2, 10))
    lam, _ = eigsolve_solver(lm, DTensor.from_numpy(scale * x0, inds), krylovdim=3, maxiter=1)
    ref, _ = ok.eigsolve_lanczos(heff(*H), x0, krylovdim=3, maxiter=1)
    assert abs(lam - ref) <= 1e-12 * abs(ref)


@pytest.mark.parametrize("precision", ["fp64", "ozaki"])
def test_waits_that_give_up(nsg_ctx, precision):
    """The cycle is repeated step by step, and nothing of it is reported by a later call."""
    rng = np.random.default_rng(3)
    lm, inds = _device_map(*_chain_heff(rng, 64, 80))
    x0 = DTensor.from_numpy(rng.standard_normal((64, 2, 2, 80)), inds)

    def solve():
        before = nsg_ctx.counters()["launches"]
        lam, x = eigsolve_solver(lm, x0, krylovdim=3, maxiter=1)
        y, info = exponentiate_solver(lm, -0.5 / abs(lam), x0, tol=1e-12)
        assert info["converged"]
        return lam, x.to_numpy(), y.to_numpy(), nsg_ctx.counters()["launches"] - before

    nsg_ctx.set_precision(precision)
    try:
        solve()  # (the exponential's next cycle starts from what the last one needed)
        lam, x, y, launches = solve()
        nsg_ctx.set_tuning("lanczos_polls", -1)
        lam_g, x_g, y_g, launches_g = solve()
        nsg_ctx.set_tuning("lanczos_polls", 0)
        assert launches_g > launches
        assert abs(lam_g - lam) <= 1e-10 * abs(lam)
        assert np.linalg.norm(x_g - x) < 1e-8 and np.linalg.norm(y_g - y) < 1e-8 * np.linalg.norm(y)
        assert abs(np.linalg.norm(x_g) - 1) < 1e-13
        nsg_ctx.set_tuning("lanczos_polls", -2)
        lam_g, x_g, _, launches_g = solve()
        nsg_ctx.set_tuning("lanczos_polls", 0)
        assert lam_g == lam and launches_g == launches
        assert np.linalg.norm(x_g - x) < 1e-14 and abs(np.linalg.norm(x_g) - 1) < 1e-13
        assert solve()[3] == launches
    finally:
        nsg_ctx.set_tuning("lanczos_polls", 0)
        nsg_ctx.set_precision("fp64")
