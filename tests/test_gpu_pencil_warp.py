"""The warp stage (two warps per pencil) against the tensor-core stage at the
edges of its loops: rows per parity class around the batches of 8 and the 32
lanes, odd and even Nx, blocks with fewer than eight pencils.  Both evaluate the
same FP64 step; bounds as in the tensor-core stage's own test (1e-12 on the
evolved fields)."""

import pytest
import torch

from jaxfun_b200.kmm import PlaneCouetteFluctuation

pytestmark = pytest.mark.gpu


def rel(a, b):
    n = float(torch.linalg.vector_norm(b))
    return float(torch.linalg.vector_norm(a - b)) / n if n else float(torch.linalg.vector_norm(a))


@pytest.mark.parametrize("N", [(9, 8, 8), (18, 6, 18), (33, 12, 16), (34, 8, 36), (64, 16, 8),
                               (65, 8, 24)])
@pytest.mark.parametrize("integrator, form, family", [
    ("SBDF3", "rotational", "C"), ("IMEXRK222", "gradient", "L")])
def test_warp_stage_matches_tensor_core_stage(cuda, N, integrator, form, family):
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
