"""The gradient on a non-blocking stream while the default stream is busy: the
buffers that the first call allocates are filled in order with the call."""

import pytest
import torch

from jaxfun_b200 import minimal_seed as ms
from jaxfun_b200.kmm import PlaneCouetteFluctuation

pytestmark = pytest.mark.gpu


def test_first_gradient_on_a_side_stream(cuda):
    def make():
        return PlaneCouetteFluctuation(N=(17, 16, 16), Re=400.0, dt=0.01,
                                       perturbation_amplitude=0.1, device=cuda,
                                       time_integrator="SBDF3", nonlinear_form="rotational")

    s, t = make(), make()
    x0 = ms._primary(s.initial_state())
    gain, grad = ms.gain_and_gradient(s, x0, 4, checkpoint=2)
    work = torch.randn(6144, 6144, device=cuda)
    torch.cuda.synchronize()
    side = torch.cuda.Stream(device=cuda)
    for _ in range(40):  # tens of milliseconds queued on the default stream
        work = torch.mm(work, work) * 1e-4
    with torch.cuda.stream(side):
        gain2, grad2 = ms.gain_and_gradient(t, x0, 4, checkpoint=2)
    torch.cuda.synchronize()
    assert gain2 == gain
    for a, b in zip((*grad.u, grad.g), (*grad2.u, grad2.g), strict=True):
        assert torch.equal(a, b)
