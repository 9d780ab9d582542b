"""First use of a space's transforms and maps on a non-blocking stream: their
operators have arrived there."""

import pytest
import torch

from jaxfun_b200.tps import TensorProductSpace

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [(257, 16, 8), (129, 24)])
def test_first_use_on_a_side_stream(cuda, N):
    dom = ((-1.0, 1.0), (0.0, 2.0), (0.0, 3.0))[:len(N)]
    order = (1,) + (0,) * (len(N) - 1)

    def run():
        T = TensorProductSpace("D", N, dom, device=cuda)
        gen = torch.Generator(device=cuda).manual_seed(1)
        c = torch.randn(T.num_dofs, generator=gen, dtype=torch.complex128, device=cuda)
        u = T.backward(c)
        return u, T.backward_primitive(c, order), T.forward(u), T.to_orthogonal(c)

    want = run()
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream(device=cuda)):
        got = run()
    torch.cuda.synchronize()
    for a, b in zip(got, want, strict=True):
        assert torch.equal(a, b)
