"""Diagonal systems through the wide-factor solve: the result is the quotient,
rounded as a division rounds it (GPU)."""

import pytest
import torch

from jaxfun_b200 import _lib
from jaxfun_b200.la import _stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 63, 130])
@pytest.mark.parametrize("dtype", [torch.float64, torch.complex128])
def test_diagonal_systems_divide(cuda, n, dtype):
    gen = torch.Generator(device=cuda).manual_seed(n)
    modes, rhs, uoffs = 500, 4, tuple(range(0, 18, 2))
    U = torch.zeros((modes, len(uoffs), n), dtype=torch.float64, device=cuda)
    U[:, 0] = torch.exp(3 * torch.randn((modes, n), generator=gen, dtype=torch.float64,
                                        device=cuda))
    b = torch.randn((rhs, n, modes), generator=gen, dtype=dtype, device=cuda)
    b[0, 0] = 0.0
    b[1, 1] = 1e-300
    x = torch.empty_like(b)
    _lib.call("jfb_wavenumber_solve", None, _lib.int64_array(()), 0, U.data_ptr(),
              _lib.int64_array(uoffs), len(uoffs), n, 1, modes, rhs, b.data_ptr(), x.data_ptr(),
              int(b.is_complex()), _stream(b))
    real = (lambda t: torch.view_as_real(t)) if b.is_complex() else (lambda t: t.unsqueeze(-1))
    want, got = real(b) / U[:, 0].T[None, :, :, None], real(x)
    # a quotient corrected by its residual may miss the rounding of a division by
    # one place in rare cases; a product with the rounded reciprocal does in a
    # quarter of them
    assert float((got != want).double().mean()) < 1e-3
    torch.testing.assert_close(got, want, rtol=2.3e-16, atol=0)
