"""Wavenumber solves with more systems than staged blocks fit on the chip: the
sizes on both sides of the rule that chooses the kernel agree with the
factors, and long systems stay in flight together (GPU)."""

import pytest
import torch

from jaxfun_b200 import _lib
from jaxfun_b200.la import _stream

pytestmark = pytest.mark.gpu

TWO_CLASSES = ((-4, -2), (0, 2, 4))
ONE_CLASS = ((-1,), (0, 1))


def _factors(offs, n, modes, cuda, gen):
    L = 0.1 * torch.randn((modes, len(offs[0]), n), generator=gen, dtype=torch.float64, device=cuda)
    U = 0.1 * torch.randn((modes, len(offs[1]), n), generator=gen, dtype=torch.float64, device=cuda)
    U[:, 0] += 4.0
    return L, U


def _solve(offs, L, U, b):
    out = torch.empty_like(b)
    rhs, n, modes = b.shape
    _lib.call("jfb_wavenumber_solve", L.data_ptr(), _lib.int64_array(offs[0]), len(offs[0]),
              U.data_ptr(), _lib.int64_array(offs[1]), len(offs[1]), n, 1, modes, rhs,
              b.data_ptr(), out.data_ptr(), int(b.is_complex()), _stream(b))
    return out


def _apply(offsets, data, x):
    """DIA product along axis 1 of (rhs, n, modes), data (modes, diagonals, n)."""
    n = x.shape[1]
    y = torch.zeros_like(x)
    for d, k in enumerate(offsets):
        if abs(k) >= n:
            continue
        cols = slice(max(0, k), min(n, n + k))
        rows = slice(max(0, -k), min(n, n - k))
        y[:, rows] += data[:, d, cols].T[None] * x[:, cols]
    return y


# chosen by the rule's lines: few and many right-hand sides of short systems,
# lengths around 24 and 64, one to several waves of blocks
@pytest.mark.parametrize("offs", [TWO_CLASSES, ONE_CLASS,
                                  ((-2,), tuple(range(0, 130, 2))),
                                  ((-3, -2, -1), tuple(range(30)))])
@pytest.mark.parametrize("n, modes, rhs", [
    (12, 600, 7), (12, 600, 8), (23, 64, 9), (24, 64, 1), (63, 2000, 2), (64, 300, 1),
    (65, 5000, 5), (129, 4096, 1), (130, 3000, 4), (255, 1000, 3)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.complex128])
def test_both_sides_of_the_kernel_rule(cuda, offs, n, modes, rhs, dtype):
    gen = torch.Generator(device=cuda).manual_seed(n + modes)
    L, U = _factors(offs, n, modes, cuda, gen)
    b = torch.randn((rhs, n, modes), generator=gen, dtype=dtype, device=cuda)
    x = _solve(offs, L, U, b)
    back = _apply(offs[1], U, x)
    back = back + _apply(offs[0], L, back)
    # backward error of two substitutions, each of at most 65 terms a row: the
    # row sums of |L| |U| are below 100 times the largest |x|
    bound = 100 * 130 * 2.3e-16 * float(x.abs().max())
    assert float((back - b).abs().max()) <= bound


def test_long_systems_stay_in_flight(cuda):
    """32768 systems of 2000 unknowns read and write 2 GB several times over: a
    few milliseconds with every vector in flight, over 80 with one staged block
    of two vectors per SM."""
    gen = torch.Generator(device=cuda).manual_seed(0)
    L, U = _factors(TWO_CLASSES, 2000, 4096, cuda, gen)
    b = torch.randn((8, 2000, 4096), generator=gen, dtype=torch.complex128, device=cuda)
    _solve(TWO_CLASSES, L, U, b)
    start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    start.record()
    _solve(TWO_CLASSES, L, U, b)
    end.record()
    end.synchronize()
    assert start.elapsed_time(end) < 30.0
