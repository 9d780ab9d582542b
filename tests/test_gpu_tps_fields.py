"""Transforms of fields with few wall-normal rows, and of fields on an 8-byte
boundary (GPU): the x operator's block size and its narrower copies."""

import ctypes
import math

import numpy as np
import pytest
import torch

from jaxfun_b200 import _lib
from jaxfun_b200.tps import TensorProductSpace
from oracle import kmm as ok

pytestmark = pytest.mark.gpu

DOM = ((-1.0, 1.0), (0.0, 4.0 * math.pi), (0.0, 2.0 * math.pi))


# round-off as in the transforms' other tests: a few eps sqrt(log2 n) per axis
@pytest.mark.parametrize("N", [(8, 32, 48), (9, 16, 128), (16, 64, 6), (17, 128, 32), (25, 18, 24),
                               (64, 16, 16)])
def test_few_rows(cuda, N):
    T = TensorProductSpace("D", N, DOM, padding_factor=(1.0, 1.5, 1.5), device=cuda)
    x = ok.Composite1D(ok.make_orthogonal("C", N[0], DOM[0]), "dirichlet")
    spaces = [x] + [ok.Fourier1D(n, d) for n, d in zip(N[1:], DOM[1:])]
    rng = np.random.default_rng(N[0])
    c = rng.standard_normal(T.num_dofs) + 1j * rng.standard_normal(T.num_dofs)
    u = c
    for ax, s in enumerate(spaces):
        u = s.backward(u, N[ax], ax)
    got = T.backward(torch.from_numpy(c).to(cuda), padded=False).cpu().numpy()
    assert np.linalg.norm(got - u) < 1e-13 * np.linalg.norm(u)


def test_field_on_an_eight_byte_boundary(cuda):
    T = TensorProductSpace("C", (17, 16, 12), DOM, device=cuda)
    gen = torch.Generator(device=cuda).manual_seed(2)
    c = torch.randn(T.num_dofs, generator=gen, dtype=torch.complex128, device=cuda)
    want = T.backward(c, padded=False)
    shifted = torch.empty(2 * c.numel() + 1, dtype=torch.float64, device=cuda)
    shifted[1:] = torch.view_as_real(c).reshape(-1)
    got = torch.empty_like(want)
    _lib.call("jfb_tps_backward", T._h, ctypes.c_void_p(shifted.data_ptr() + 8), got.data_ptr(), 0,
              ctypes.c_void_p(torch.cuda.current_stream(cuda).cuda_stream))
    assert torch.equal(got, want)
