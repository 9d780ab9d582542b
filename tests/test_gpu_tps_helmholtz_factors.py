"""The fused Helmholtz solve with factors of every form its entry takes, without
explicit inverses: L offsets other than -2 and -4, odd offsets, and factors
beyond shared memory, against dense solves between the separate transforms."""

import numpy as np
import pytest
import torch

from jaxfun_b200 import _lib
from jaxfun_b200.tps import Helmholtz2D, _stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N, loffs, uoffs", [
    ((16, 8), (), (0,)),
    ((16, 8), (-3, -1), (0, 1, 2, 5)),
    ((40, 6), (-4, -2), tuple(range(0, 38, 2))),
    ((67, 12), (-2,), tuple(range(40))),       # several diagonals per lane
    ((100, 8), (-2,), tuple(range(42))),       # 47 KB with the kernel's own 2 KB: over 48
    ((131, 4), (-6, -4, -2), (0, 2, 128)),
    ((160, 2), (-1,), tuple(range(158))),      # 201 KB of factors: read from memory
])
def test_general_factors(cuda, N, loffs, uoffs):
    h = Helmholtz2D(N, device=cuda)
    assert h.fused
    n, m = h.TD.num_dofs[0], N[1]
    rng = np.random.default_rng(N[0])
    # rows of |L - I| and |U - diag| sum to about one against a diagonal of three
    L = rng.standard_normal((m, len(loffs), n)) * 0.3
    U = rng.standard_normal((m, len(uoffs), n)) / len(uoffs)
    U[:, 0] = 3.0 + rng.random((m, n))
    lower, upper = np.zeros((2, m, n, n))
    lower += np.eye(n)
    for offs, data, dense in ((loffs, L, lower), (uoffs, U, upper)):
        for d, off in enumerate(offs):
            for col in range(max(0, off), min(n, n + off)):
                dense[:, col - off, col] = data[:, d, col]
    f = torch.from_numpy(rng.standard_normal(N) + 1j * rng.standard_normal(N)).to(cuda)
    tl, tu = (torch.from_numpy(v).to(cuda) for v in (L, U))
    u = torch.empty(h.TD.N, dtype=torch.complex128, device=cuda)
    _lib.call("jfb_helmholtz2d_solve", h.TC._h, h.TD._h, tl.data_ptr() if loffs else None,
              _lib.int64_array(loffs), len(loffs), tu.data_ptr(), _lib.int64_array(uoffs),
              len(uoffs), None, h._fourier_mass, f.data_ptr(), u.data_ptr(), _stream(cuda))
    rhs = (h.TD.scalar_product(h.TC.backward(f)) / h._fourier_mass).cpu().numpy()
    sol = np.linalg.solve(lower @ upper, rhs.T[:, :, None])[:, :, 0].T
    want = h.TD.backward(torch.from_numpy(sol.copy()).to(cuda)).cpu().numpy()
    # both sides solve modes of condition below 100 and transform: the bound of
    # the fused solve's other tests
    assert np.linalg.norm(u.cpu().numpy() - want) < 1e-12 * np.linalg.norm(want)
