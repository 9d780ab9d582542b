"""Fields that the one-launch Kronecker sum leaves to the general path (CPU:
shapes only, nothing is computed)."""

import pytest
import torch

from jaxfun_b200.la import DiaMatrix, TPMatrix, _fused_sum


def _dia(n, offsets):
    return DiaMatrix(torch.empty((len(offsets), n), dtype=torch.float64, device="meta"), offsets,
                     (n, n))


@pytest.mark.parametrize("shape, diagonals, terms", [
    ((3, 1 << 16, 1 << 16), 2, 1),     # more modes than a 32-bit index holds
    ((257, 64, 64), 129, 1),           # long dense operators on few modes
    ((64, 257, 64), 129, 3),
    ((800, 4, 4), 3, 1),               # a column block beyond shared memory
])
def test_left_to_the_general_path(shape, diagonals, terms):
    poly = shape.index(max(shape)) if shape[0] != 3 else 0
    mats = [_dia(n, tuple(range(0, 2 * diagonals, 2)) if a == poly else (0,))
            for a, n in enumerate(shape)]
    u = torch.empty(shape, dtype=torch.complex128, device="meta")
    assert _fused_sum([TPMatrix(mats, 1.0)] * terms, u) is None
