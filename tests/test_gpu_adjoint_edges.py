"""The reverse sweep at the edges of its kernels: odd and even Nx, both record
layouts (Nx <= 65 and above), whole and partial tiles of wavenumbers, one and two
row tiles per warp (above Nx = 67), periodic lengths with and without a
warp-shuffle transform, and segments of one to several steps (GPU).

The directional derivative against central differences with eps = 1e-5: their
truncation is of order eps^2, and the gain's round-off (a few 1e-15) divided by
2 eps is 2e-10, which the absolute bound allows for; the relative one is that of
the adjoint's own tests."""

import pytest

from jaxfun_b200 import minimal_seed as ms
from jaxfun_b200.kmm import PlaneCouetteFluctuation
from jaxfun_b200.workloads import couette_perturbation_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N, steps", [
    ((18, 16, 16), 4),   # even Nx, 24-point lines
    ((33, 64, 12), 5),   # 96-point y lines, 18-point z lines
    ((16, 12, 64), 6),   # 96-point z lines
    ((65, 8, 64), 4),    # largest one-kernel tile
    ((67, 16, 8), 4),    # block records, half a kz tile
    ((80, 64, 24), 4),   # even Nx with block records, ragged kz tiles, 96-point y lines
    ((129, 8, 64), 4),   # largest Nx: two row tiles per warp, 96-point z lines
])
def test_gradient_at_size_edges(cuda, N, steps):
    s = PlaneCouetteFluctuation(N=N, Re=400.0, dt=0.01, perturbation_amplitude=0.1, device=cuda,
                                time_integrator="SBDF3", nonlinear_form="rotational")
    x0 = ms._primary(s.initial_state())
    f = couette_perturbation_fields(s.N, s.domain, seeds=(200, 201))
    d = ms._primary(s.state_from_physical(f))
    d = ms.tree_scale(d, ms.tree_l2_norm(x0) / ms.tree_l2_norm(d))
    eps = 1e-5
    jp = ms.perturbation_gain(s, ms.tree_add_scaled(x0, d, eps), steps)
    jm = ms.perturbation_gain(s, ms.tree_add_scaled(x0, d, -eps), steps)
    fd = (jp - jm) / (2 * eps)
    values = []
    for stride in (1, 3, steps):  # segments of one step, a ragged last one, one segment
        _, g = ms.gain_and_gradient(s, x0, steps, checkpoint=stride)
        values.append(ms.jax_complex_directional_derivative(g, d))
    for v in values:
        assert abs(v - fd) <= 1e-6 * abs(fd) + 2e-10
        assert abs(v - values[0]) <= 1e-12 * abs(values[0]) + 1e-15
