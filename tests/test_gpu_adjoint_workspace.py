"""Device memory of the gradient's reverse sweep: a run for the gain alone takes
none, the kept buffers are counted and serve later calls that need no more."""

import pytest
import torch

from jaxfun_b200 import minimal_seed as ms
from jaxfun_b200.kmm import PlaneCouetteFluctuation

pytestmark = pytest.mark.gpu


def _free(device):
    """Device memory that neither the library nor the process's context holds."""
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(device)[0] + torch.cuda.memory_reserved(device)


def test_sweep_buffers_are_allocated_for_gradients_only(cuda):
    s = PlaneCouetteFluctuation(N=(33, 32, 32), Re=400.0, dt=0.01, perturbation_amplitude=0.1,
                                device=cuda, time_integrator="SBDF3",
                                nonlinear_form="rotational")
    x0 = ms._primary(s.initial_state())
    ms.perturbation_gain(s, x0, 3)  # operators uploaded, kernels loaded
    free, held = _free(cuda), s.info().device_bytes
    gain = ms.perturbation_gain(s, x0, 40)
    assert _free(cuda) == free and s.info().device_bytes == held
    # six fields of 16 bytes per (x, ky, kz >= 0) and step of a segment
    fields = 96 * 33 * 32 * 16
    value, grad = ms.gain_and_gradient(s, x0, 40, checkpoint=10)
    kept = s.info().device_bytes - held
    assert value == gain and kept >= 10 * fields
    assert free - _free(cuda) >= 10 * fields
    # shorter runs and segments, and gains in between, find the buffers there
    free = _free(cuda)
    for steps, checkpoint in ((40, 10), (17, 6), (3, 20), (40, 10)):
        ms.perturbation_gain(s, x0, 5)
        again = ms.gain_and_gradient(s, x0, steps, checkpoint=checkpoint)[1]
        assert _free(cuda) == free and s.info().device_bytes - held == kept
    for a, b in zip((*grad.u, grad.g), (*again.u, again.g), strict=True):
        assert torch.equal(a, b)
