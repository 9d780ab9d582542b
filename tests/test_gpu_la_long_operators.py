"""Kronecker sums on both sides of the rule that sends long dense operators on
few modes to the general path (GPU)."""

import pytest
import torch

from jaxfun_b200.la import DiaMatrix, TPMatrices, TPMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape, poly, diagonals", [
    ((130, 6, 5), 0, 65), ((5, 180, 4), 1, 88), ((6, 5, 200), 2, 100), ((257, 12), 0, 129),
    ((150, 100, 90), 0, 110)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.complex128])
def test_sum_equals_its_terms(cuda, shape, poly, diagonals, dtype):
    gen = torch.Generator(device=cuda).manual_seed(sum(shape))

    def dia(n, offsets):
        return DiaMatrix(torch.randn((len(offsets), n), generator=gen, dtype=torch.float64,
                                     device=cuda), offsets, (n, n))

    op = TPMatrices([TPMatrix([dia(n, tuple(range(0, 2 * diagonals, 2)) if a == poly else (0,))
                               for a, n in enumerate(shape)], c) for c in (1.0, -0.5)])
    u = torch.randn(shape, generator=gen, dtype=dtype, device=cuda)
    got, want = op @ u, sum(tp @ u for tp in op.tpmats)
    # sums of at most 130 products of normal numbers in two orders
    assert float((got - want).abs().max()) <= 2 * 130 * 2.3e-16 * 130 * float(want.abs().max())
