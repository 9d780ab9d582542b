"""The gradient with outputs left out: each array that is asked for is that of
the full call, and a call that asks for none still returns the gain."""

import ctypes

import pytest
import torch

from jaxfun_b200 import _lib
from jaxfun_b200 import minimal_seed as ms
from jaxfun_b200.kmm import PlaneCouetteFluctuation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaves", [(), ("g",), ("u0", "u2")])
def test_gradient_with_null_outputs(cuda, leaves):
    s = PlaneCouetteFluctuation(N=(17, 16, 16), Re=400.0, dt=0.01, perturbation_amplitude=0.1,
                                device=cuda, time_integrator="SBDF3",
                                nonlinear_form="rotational")
    x0 = ms._primary(s.initial_state())
    gain, full = ms.gain_and_gradient(s, x0, 3)
    want = {"u0": full.u[0], "u1": full.u[1], "u2": full.u[2], "g": full.g}
    out = {k: torch.empty_like(want[k]) for k in leaves}
    c = _lib.KMMStateC()
    for k, v in out.items():
        setattr(c, k, v.data_ptr())
    value = ctypes.c_double()
    _lib.call("jfb_kmm_gain_gradient", s._plan, ctypes.byref(ms._c(s, x0)), 3, 20,
              ctypes.byref(value), ctypes.byref(c), s._stream())
    assert value.value == gain
    for k, v in out.items():
        assert torch.equal(v, want[k])
