"""The FP64 products' small-tile and tall-skinny kernels at the sizes where they can go
wrong: edges of the 16 x 16 tiles, remainders of the K slabs and of the K slices, batches,
every orientation and conjugation, against numpy in the same precision.  Tolerance: a
product of depth K summed in any order is within K eps of the absolute product."""
import numpy as np
import pytest

from networksolvers_gb300.itensors import DTensor, Index, contract

pytestmark = pytest.mark.gpu


def rnd(rng, shape, cplx):
    x = rng.standard_normal(shape)
    return x + 1j * rng.standard_normal(shape) if cplx else x


def close(got, ref, mag, k):
    assert np.all(np.abs(got - ref) <= 4 * (k + 4) * 2.3e-16 * mag + 1e-300)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n,k", [(1, 40, 1), (15, 33, 31), (16, 48, 32), (17, 35, 33), (40, 64, 257), (64, 64, 126),
                                   (33, 100, 15), (130, 90, 64), (700, 41, 19), (300, 290, 70)])
def test_tile_products_every_orientation(nsg_ctx, cplx, m, n, k):
    rng = np.random.default_rng(m + 7 * n + 31 * k)
    a, b = rnd(rng, (m, k), cplx), rnd(rng, (k, n), cplx)
    mag = np.abs(a) @ np.abs(b)
    i, j, l = Index(m), Index(n), Index(k)
    for ta in (False, True):
        A = DTensor.from_numpy(a.T, [l, i]) if ta else DTensor.from_numpy(a, [i, l])
        for tb in (False, True):
            B = DTensor.from_numpy(b.T, [j, l]) if tb else DTensor.from_numpy(b, [l, j])
            close(contract([A, B], out=[i, j]).to_numpy(), a @ b, mag, k)
            close(contract([A, B], out=[j, i]).to_numpy(), (a @ b).T, mag.T, k)
            if cplx:
                close(contract([A.dag(), B], out=[i, j]).to_numpy(), a.conj() @ b, mag, k)
                close(contract([A, B.dag()], out=[i, j]).to_numpy(), a @ b.conj(), mag, k)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n,k,batch", [(20, 36, 40, 3), (16, 64, 64, 37), (65, 40, 33, 5)])
def test_tile_products_batched(nsg_ctx, cplx, m, n, k, batch):
    rng = np.random.default_rng(m + batch)
    a, b = rnd(rng, (m, k, batch), cplx), rnd(rng, (k, n), cplx)
    i, j, l, q = Index(m), Index(n), Index(k), Index(batch)
    got = contract([DTensor.from_numpy(a, [i, l, q]), DTensor.from_numpy(b, [l, j])], out=[i, j, q]).to_numpy()
    close(got, np.einsum("ilq,lj->ijq", a, b), np.einsum("ilq,lj->ijq", np.abs(a), np.abs(b)), k)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n,k,batch", [(1, 1, 1, 1), (3, 5, 7, 50), (64, 20, 20, 64), (6, 32, 32, 11), (257, 12, 20, 3),
                                         (300, 20, 12, 200)])
def test_skinny_products(nsg_ctx, cplx, m, n, k, batch):
    """op(B) mixes zeros, powers of two (of both signs) and general values, as operator
    tensors do; batch entries shorter and longer than a CTA's rows."""
    rng = np.random.default_rng(m + 5 * batch)
    a, b = rnd(rng, (m, k, batch), cplx), rnd(rng, (k, n), cplx)
    kind = rng.integers(0, 4, (k, n))
    b = np.where(kind == 0, 0.0, np.where(kind == 1, 2.0 ** rng.integers(-3, 4, (k, n)) * rng.choice([-1, 1], (k, n)), b))
    i, j, l, q = Index(m), Index(n), Index(k), Index(batch)
    for t in (False, True):
        B = DTensor.from_numpy(b.T, [j, l]) if t else DTensor.from_numpy(b, [l, j])
        got = contract([DTensor.from_numpy(a, [i, l, q]), B], out=[i, j, q]).to_numpy()
        close(got, np.einsum("ilq,lj->ijq", a, b), np.einsum("ilq,lj->ijq", np.abs(a), np.abs(b)), k)


def test_skinny_power_of_two_terms_are_exact(nsg_ctx):
    """A column with one power-of-two entry is that multiple of A's column, bit for bit, at
    the ends of the exponent range too (zeros, subnormals, the largest numbers)."""
    rng = np.random.default_rng(3)
    a = rng.standard_normal((64, 4)) * 10.0 ** rng.integers(-307, 307, (64, 4))
    a[:6, 0] = [0.0, 5e-324, -2.3e-308, 1.7e308, -1.7e308, 1.0]
    b = np.zeros((4, 6))
    b[0, 0], b[0, 1], b[0, 2], b[1, 3], b[2, 4], b[3, 5] = 1.0, -0.5, 2.0 ** -40, 4.0, -1.0, 2.0 ** 300
    i, j, l = Index(64), Index(6), Index(4)
    got = contract([DTensor.from_numpy(a, [i, l]), DTensor.from_numpy(b, [l, j])], out=[i, j]).to_numpy()
    with np.errstate(over="ignore", under="ignore"):
        ref = np.stack([a[:, r] * b[r, c] for c, r in enumerate([0, 0, 0, 1, 2, 3])], 1)
    assert np.array_equal(got, ref)
