"""The wavenumber solve at its smallest systems: one unknown (a single parity
class) and two (one unknown per class, or coupled), for factors with few and
with many diagonals, several modes and right-hand sides (GPU)."""

import numpy as np
import pytest
import torch

from jaxfun_b200 import _lib
from jaxfun_b200.la import DiaMatrix, _stream

pytestmark = pytest.mark.gpu

# (L offsets, U offsets): diagonals past the last column hold nothing
FACTORS = {
    "diagonal": ((), (0,)),
    "even": ((-4, -2), (0, 2, 4)),
    "coupled": ((-1,), (0, 1)),
    "wide": ((-2, -1), tuple(range(9))),
}


@pytest.mark.parametrize("factors", FACTORS)
@pytest.mark.parametrize("n", [1, 2])
@pytest.mark.parametrize("outer, inner", [(1, 1), (1, 7), (5, 1), (3, 40)])
@pytest.mark.parametrize("rhs, cplx", [(1, False), (3, True), (9, True)])
def test_one_and_two_unknowns(cuda, factors, n, outer, inner, rhs, cplx):
    loffs, uoffs = FACTORS[factors]
    rng = np.random.default_rng(n + 10 * outer + rhs)
    modes = outer * inner
    L = 0.2 * rng.standard_normal((modes, len(loffs), n))
    U = 0.2 * rng.standard_normal((modes, len(uoffs), n))
    U[:, 0, :] += 4.0
    lower, upper = np.zeros((2, modes, n, n))
    lower += np.eye(n)
    for offs, data, dense in ((loffs, L, lower), (uoffs, U, upper)):
        for d, off in enumerate(offs):
            for col in range(max(0, off), min(n, n + off)):
                dense[:, col - off, col] = data[:, d, col]
    b = rng.standard_normal((rhs, outer, n, inner))
    if cplx:
        b = b + 1j * rng.standard_normal(b.shape)
    tl, tu, tb = (torch.from_numpy(v).to(cuda) for v in (L, U, b))
    # a guard band after the result shows a write past its end
    flat = torch.full((tb.numel() + 64,), 7.0, dtype=tb.dtype, device=cuda)
    _lib.call("jfb_wavenumber_solve", tl.data_ptr() if loffs else None, _lib.int64_array(loffs),
              len(loffs), tu.data_ptr(), _lib.int64_array(uoffs), len(uoffs), n, outer, inner, rhs,
              tb.data_ptr(), flat.data_ptr(), int(cplx), _stream(tb))
    assert bool((flat[tb.numel():] == 7.0).all())
    got = flat[:tb.numel()].reshape(tb.shape).cpu().numpy()
    cols = np.moveaxis(b, 2, 3).reshape(rhs, modes, n).transpose(1, 2, 0)
    ref = np.linalg.solve(lower @ upper, cols).transpose(2, 0, 1).reshape(rhs, outer, inner, n)
    # at most two unknowns, condition below 10 on both sides of the comparison
    np.testing.assert_allclose(got, np.moveaxis(ref, 3, 2), rtol=0,
                               atol=64 * 2.3e-16 * max(1.0, np.abs(ref).max()))


def test_solve_of_a_one_by_one_matrix(cuda):
    A = DiaMatrix.from_dense(torch.tensor([[4.0]], dtype=torch.float64, device=cuda))
    b = torch.arange(1.0, 131.0, dtype=torch.float64, device=cuda).reshape(1, 130)
    torch.testing.assert_close(A.solve(b), b / 4.0, rtol=0, atol=0)
