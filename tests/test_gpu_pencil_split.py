"""The two-kernel pencil stage (Nx above the one-kernel tile) against the
warp-per-pencil stage: edge sizes of its tiles (rows, pencils, odd and even
Nx), every integrator (with and without a linear term), both forms and
families.  Both evaluate the same FP64 step: the bounds are those of the
one-kernel stage's test (1e-12 on the evolved fields, 1e-10 on history rows,
whose operators amplify rounding by Nx^2)."""

import pytest
import torch

from jaxfun_b200.kmm import PlaneCouetteFluctuation

pytestmark = pytest.mark.gpu


def rel(a, b):
    n = float(torch.linalg.vector_norm(b))
    return float(torch.linalg.vector_norm(a - b)) / n if n else float(torch.linalg.vector_norm(a))


@pytest.mark.parametrize("N", [(67, 16, 16), (80, 8, 18), (97, 24, 8), (128, 12, 16), (129, 6, 36)])
@pytest.mark.parametrize("integrator, form, family", [
    ("SBDF3", "rotational", "C"), ("CNAB2", "gradient", "C"), ("IMEXRK222", "rotational", "L"),
    ("IMEXRK3", "gradient", "L")])
def test_split_stage_matches_warp_stage(cuda, N, integrator, form, family):
    def make():
        return PlaneCouetteFluctuation(N=N, Re=1000.0, dt=0.01, perturbation_amplitude=0.02,
                                       device=cuda, time_integrator=integrator,
                                       nonlinear_form=form, family=family)

    g1, g2 = make(), make()
    assert g1.variant()["current"]["pencil"] == 1
    g2.set_variant(pencil=0)
    s0 = g1.initial_state()
    a, b = g1.solve(s0, 5), g2.solve(s0, 5)
    for x, y in zip((*a.u, a.g), (*b.u, b.g), strict=True):
        assert rel(x, y) < 1e-12
    if integrator == "SBDF3":
        for x, y in zip(a.nonlinear_old, b.nonlinear_old, strict=True):
            assert rel(x, y) < 1e-10
