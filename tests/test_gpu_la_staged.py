"""The staged wavenumber solve and the fused Kronecker product against dense
algebra, at the edges of their blocks (modes, right-hand sides, rows) and on
both layouts (polynomial axis first, in the middle, last)."""

import itertools

import numpy as np
import pytest
import torch

from jaxfun_b200.la import DiaMatrix, TPMatrices, TPMatrix, tpmats_wavenumber_factor

pytestmark = pytest.mark.gpu


def _banded(n, offsets, rng):
    a = np.zeros((n, n))
    for k in offsets:
        if abs(k) < n:
            a += np.diag(rng.standard_normal(n - abs(k)) * 0.2, k)
    return a + 4 * np.eye(n)


def _operator(shape, poly, offsets, rng, dev):
    """Two terms A (x) ones + B (x) Fourier weights, and their dense per-mode sums."""
    n = shape[poly]
    A, B = _banded(n, offsets, rng), _banded(n, offsets, rng)
    four = [a for a in range(len(shape)) if a != poly]
    w = [1.0 + 0.1 * rng.random(shape[a]) for a in four]
    offs = [k for k in offsets if abs(k) < n]
    dia = {id(m): DiaMatrix.from_dense(torch.from_numpy(m).to(dev), offs) for m in (A, B)}

    def term(m, ws, coef):
        mats = [None] * len(shape)
        mats[poly] = dia[id(m)]
        for a, v in zip(four, ws):
            mats[a] = DiaMatrix(torch.from_numpy(v[None].copy()).to(dev), (0,), (v.size, v.size))
        return TPMatrix(mats, coef)

    ones = [np.ones(shape[a]) for a in four]
    W = w[0] if len(w) == 1 else np.multiply.outer(w[0], w[1])
    dense = A + 0.5 * W.reshape(-1, 1, 1) * B  # (modes, n, n)
    return TPMatrices([term(A, ones, 1.0), term(B, w, 0.5)]), dense


WIDE_EVEN = (-2, *range(0, 60, 2))
WIDE_ODD = (-3, -1, *range(0, 31))
NARROW_EVEN = (-4, -2, 0, 2, 4)
NARROW_ODD = (-1, 0, 1)


@pytest.mark.parametrize("offsets", [WIDE_EVEN, WIDE_ODD, NARROW_EVEN, NARROW_ODD])
@pytest.mark.parametrize("shape, poly", [((5, 3), 0), ((33, 6, 5), 0), ((4, 64, 3), 1),
                                         ((7, 5, 65), 2), ((97, 17), 0), ((9, 127), 1)])
@pytest.mark.parametrize("rhs, cplx", [(1, True), (3, False), (9, True)])
def test_solve_and_product_match_dense(cuda, offsets, shape, poly, rhs, cplx):
    rng = np.random.default_rng(len(offsets) + shape[0] + rhs)
    op, dense = _operator(shape, poly, offsets, rng, cuda)
    b = rng.standard_normal((rhs, *shape))
    if cplx:
        b = b + 1j * rng.standard_normal(b.shape)
    x = tpmats_wavenumber_factor(op).solve_many(torch.from_numpy(b).to(cuda)).cpu().numpy()
    n = shape[poly]
    cols = np.moveaxis(b, poly + 1, -1).reshape(rhs, -1, n).transpose(1, 2, 0)
    ref = np.linalg.solve(dense, cols)
    got = np.moveaxis(x, poly + 1, -1).reshape(rhs, -1, n).transpose(1, 2, 0)
    # the matrices are diagonally dominant (condition < 50): n rounding errors each
    np.testing.assert_allclose(got, ref, rtol=0, atol=50 * n * 2.3e-16 * np.abs(ref).max())
    y = (op @ torch.from_numpy(b[0]).to(cuda)).cpu().numpy()
    want = np.moveaxis((dense @ cols[:, :, :1])[:, :, 0].reshape(
        *(s for a, s in enumerate(shape) if a != poly), n), -1, poly)
    np.testing.assert_allclose(y, want, rtol=0, atol=4 * n * 2.3e-16 * np.abs(want).max())


def test_fused_product_equals_the_factors_one_by_one(cuda):
    """The fused sum against the general path (one product per factor)."""
    rng = np.random.default_rng(1)
    for shape, poly in itertools.product([(8, 6, 10), (6, 12)], (0, 1)):
        op, _ = _operator(shape, poly, (-1, 0, 2), rng, cuda)
        u = torch.from_numpy(rng.standard_normal(shape)).to(cuda)
        for v in (u, u.to(torch.float32), torch.complex(u, -u).transpose(0, 1).contiguous()
                  .transpose(0, 1)):
            want = sum(tp @ v for tp in op.tpmats)
            got = op @ v
            assert got.dtype == want.dtype and got.shape == want.shape
            torch.testing.assert_close(got, want, rtol=0, atol=1e-14 * float(want.abs().max()))
    with pytest.raises(ValueError):
        op @ u[:-1]
