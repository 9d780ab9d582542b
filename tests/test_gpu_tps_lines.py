"""Transform kernels at the edges of their size rules against the oracle, and
the fused Helmholtz solve against the separate launches (GPU)."""

import math

import numpy as np
import pytest
import torch

from jaxfun_b200.tps import Helmholtz2D, TensorProductSpace
from oracle import kmm as ok

pytestmark = pytest.mark.gpu

DOM = ((-1.0, 1.0), (0.0, 4.0 * math.pi), (0.0, 2.0 * math.pi))


def rel(a, b):
    a = a.detach().cpu().numpy()
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


# Round-off of the x product (<= 130 terms) and two transforms of <= 1296
# points: a few eps sqrt(log2 n) each, far below 1e-13 relative in the L2 norm;
# the Dirichlet forward solves with a mass of condition up to 4 N^2.
@pytest.mark.parametrize("basis,N", [
    ("C", (9, 64, 64)),     # one k tile and a remainder; 96-point warp lines
    ("D", (66, 64, 6)),     # few columns in the middle axis: Stockham
    ("C", (130, 96, 8)),    # 144-point Stockham / 96-point warp lines
    ("D", (16, 128, 128)),  # 128 and 192 points
    ("C", (17, 96)),        # 2-D: middle axis contiguous
    ("D", (12, 864)),       # 2-D, long lines: fewer of them per block
    ("C", (8, 2)),          # smallest
])
@pytest.mark.parametrize("padded", [False, True])
def test_transforms_at_size_edges(cuda, basis, N, padded):
    pad = (1.0,) + (1.5,) * (len(N) - 1)
    if padded and N[1] == 2:
        pad = (1.0, 2.0)
    T = TensorProductSpace(basis, N, DOM[:len(N)], padding_factor=pad, device=cuda)
    orth = ok.make_orthogonal("C", N[0], DOM[0])
    x = orth if basis == "C" else ok.Composite1D(orth, "dirichlet" if basis == "D" else "biharmonic")
    spaces = [x] + [ok.Fourier1D(n, d) for n, d in zip(N[1:], DOM[1:])]
    counts = [int(p * n) if padded else n for p, n in zip(pad, N)]
    rng = np.random.default_rng(11)
    c = rng.standard_normal(T.num_dofs) + 1j * rng.standard_normal(T.num_dofs)
    u = c
    for ax, s in enumerate(spaces):
        u = s.backward(u, counts[ax], ax)
    assert rel(T.backward(torch.from_numpy(c).to(cuda), padded=padded), u) < 1e-13
    v = rng.standard_normal(counts) + 1j * rng.standard_normal(counts)
    f = v
    for ax in reversed(range(len(N))):
        f = spaces[ax].forward(f, ax)
    tol = 1e-13 if basis == "C" else 1e-13 + 2.2e-16 * 4 * N[0] ** 2
    assert rel(T.forward(torch.from_numpy(v).to(cuda), padded=padded), f) < tol


# Both sides are FP64 solves of the same well-conditioned modes; 1e-12 leaves
# a factor of 30 over eps N for the largest N here.
@pytest.mark.parametrize("N", [(8, 2), (16, 1296), (130, 16), (131, 16), (150, 16), (67, 54)])
def test_helmholtz2d_fused_sizes(cuda, N):
    h = Helmholtz2D(N, device=cuda)
    assert h.fused
    rng = np.random.default_rng(3)
    f = torch.from_numpy(rng.standard_normal(N) + 1j * rng.standard_normal(N)).to(cuda)
    sep = h.separate(f).cpu().numpy()
    assert rel(h(f), sep) < 1e-12
    h._Uinv = None
    assert rel(h(f), sep) < 1e-12
