"""The work whose speed is measured: plane-Couette programs through the public API.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges,
``prepare(case, seed)`` builds what a program holds before the call (solver,
state, operators), ``run(state)`` is one pass through the public entry points,
``work(case)`` the bytes and operations the pass cannot do without, and
``exact(case, seed)`` the same results from plain torch in 64 bits (dense
x-operators and per-wavenumber inverses, full complex spectra).

Kinds:

* ``flow``      blocks of ``KMM.solve`` with the diagnostics of the block's end,
                as the cadence loop of a production run calls them; one ``step``
                at a time for ``steps = 1``;
* ``mhd``       the coupled flow + vector-potential solver, the same loop;
* ``ensemble``  independent MHD members of uneven wall-normal size;
* ``seed``      perturbation gain and its gradient (the minimal-seed ascent's
                inner call: forward sweep, checkpoints, reverse sweep);
* ``helmholtz`` the 2-D Helmholtz solve;
* ``transform`` padded backward and forward transforms of a tensor-product
                space, and a padded derivative;
* ``kron``      a Kronecker operator applied to a field and its per-wavenumber
                solve for several right-hand sides.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from jaxfun_b200.kmm import KMMState, PlaneCouetteFluctuation
from jaxfun_b200.la import DiaMatrix, TPMatrices, TPMatrix, tpmats_wavenumber_factor
from jaxfun_b200.mhd import Ensemble, MHDState, PlaneCouetteMHD
from jaxfun_b200.minimal_seed import gain_and_gradient
from jaxfun_b200.tps import Helmholtz2D, TensorProductSpace

DOMAIN = ((-1.0, 1.0), (0.0, 4.0 * math.pi), (0.0, 2.0 * math.pi))
WARM = 3  # steps taken before the timed block: a developed state with its history


def listed():
    def flow(name, n, steps, integrator="SBDF3", form="rotational", family="C", precision="fp64"):
        return {"name": name, "kind": "flow", "nx": n[0], "ny": n[1], "nz": n[2], "steps": steps,
                "integrator": integrator, "form": form, "family": family, "precision": precision}

    return [
        # the solver as its constructor's defaults build it, stepped from a
        # user's own loop: the smallest grid, where launches are everything
        flow("default_step_17", (17, 16, 16), 1, "IMEXRK222", "gradient"),
        # a ragged grid (padded lengths 24 and 72) with the Legendre family
        flow("ragged_legendre_33", (33, 16, 48), 10, "CNAB2", "gradient", "L"),
        # the production grid, both forms: blocks of 25 steps
        flow("couette_65_fp64", (65, 64, 64), 25),
        flow("couette_65_mixed", (65, 64, 64), 25, precision="mixed"),
        # the larger grids of the resolution study
        flow("couette_97_fp64", (97, 96, 96), 10),
        flow("couette_129_mixed", (129, 128, 128), 10, precision="mixed"),
        # MHD Couette flow at the production grid
        {"name": "mhd_65_fp64", "kind": "mhd", "nx": 65, "ny": 64, "nz": 64, "steps": 10,
         "precision": "fp64"},
        # a sweep's members, two of each wall-normal size, stepped together
        {"name": "ensemble_6_mixed", "kind": "ensemble", "nx": 33, "nx2": 49, "nx3": 65,
         "ny": 64, "nz": 64, "members": 6, "steps": 10, "precision": "mixed"},
        # one gradient of the minimal-seed ascent
        {"name": "seed_gradient_65", "kind": "seed", "nx": 65, "ny": 64, "nz": 64, "steps": 40,
         "checkpoint": 20},
        # the 2-D model problem: latency of a single small solve
        {"name": "helmholtz_64", "kind": "helmholtz", "nx": 64, "ny": 64},
        # dealiased transforms of a velocity component
        {"name": "transform_65", "kind": "transform", "basis": "D", "family": "C", "nx": 65,
         "ny": 64, "nz": 64, "padded": True},
        # implicit operator and solve of a user's own time stepper
        {"name": "kron_65", "kind": "kron", "family": "C", "nx": 65, "ny": 64, "nz": 64,
         "rhs": 3},
    ]


_PERIODIC = (16, 24, 32, 48, 64, 72, 96, 128)


def _grid(rng, nx_max, cost_max):
    while True:
        nx = int(round(math.exp(rng.uniform(math.log(9), math.log(nx_max)))))
        ny, nz = rng.choice(_PERIODIC), rng.choice(_PERIODIC)
        if nx * ny * nz <= cost_max:
            return nx, ny, nz


def draw(rng):
    kind = rng.choice(("flow", "flow", "flow", "flow", "mhd", "ensemble", "seed", "helmholtz",
                       "transform", "kron"))
    if kind == "flow":
        nx, ny, nz = _grid(rng, 129, 129 * 128 * 128)
        integrator = rng.choice(("SBDF3", "SBDF3", "SBDF3", "IMEXRK222", "IMEXRK3", "CNAB2"))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": rng.randint(1, 10),
                "integrator": integrator, "form": rng.choice(("rotational", "gradient")),
                "family": rng.choice("CCL"), "precision": rng.choice(("fp64", "mixed"))}
    if kind == "mhd":
        nx, ny, nz = _grid(rng, 65, 65 * 64 * 64)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": rng.randint(1, 10),
                "precision": rng.choice(("fp64", "mixed"))}
    if kind == "ensemble":
        sizes = [rng.randint(17, 65) for _ in range(3)]
        return {"kind": kind, "nx": sizes[0], "nx2": sizes[1], "nx3": sizes[2],
                "ny": rng.choice((32, 48, 64)), "nz": rng.choice((16, 32, 48, 64)),
                "members": rng.randint(2, 6), "steps": rng.randint(1, 10),
                "precision": rng.choice(("fp64", "mixed"))}
    if kind == "seed":
        nx, ny, nz = _grid(rng, 65, 65 * 64 * 64)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": rng.randint(3, 30),
                "checkpoint": rng.randint(2, 20)}
    if kind == "helmholtz":
        return {"kind": kind, "nx": rng.randint(16, 100), "ny": rng.choice((16, 24, 32, 48, 64, 96))}
    if kind == "transform":
        nx, ny, nz = _grid(rng, 129, 129 * 96 * 96)
        return {"kind": kind, "basis": rng.choice("CDB"), "family": rng.choice("CL"), "nx": nx,
                "ny": ny, "nz": nz, "padded": rng.random() < 0.7}
    nx, ny, nz = _grid(rng, 129, 97 * 96 * 96)
    return {"kind": kind, "family": rng.choice("CL"), "nx": nx, "ny": ny, "nz": nz,
            "rhs": rng.randint(1, 4)}


# -- inputs --------------------------------------------------------------------


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed, salt=0):
    return torch.Generator().manual_seed(1_000_003 * int(seed) + salt)


def _dt(case):
    """Time step of the benchmark workload."""
    return 0.01


def _re(case):
    return 1000.0


def _nodes(family, n):
    if family == "L":
        return np.polynomial.legendre.leggauss(n)[0]
    return np.cos(np.pi + (2 * np.arange(n) + 1) * np.pi / (2 * n))


def _velocity(nx, ny, nz, family, seed, dev):
    """Divergence-free perturbation curl(psi_a e_z) + curl(psi_b e_y),
    psi = (1 - x^2)^2 sum_k w_k [alpha cos k.y + beta sin k.y],
    w = exp(-|k|^2 / 16), |k| up to a third of the modes, at energy 1e-4."""
    x = torch.from_numpy(_nodes(family, nx)).to(dev)
    env, denv = (1 - x**2) ** 2, -4 * x * (1 - x**2)
    my, mz = ny // 3, nz // 3
    ky, kz = torch.arange(-my, my + 1), torch.arange(-mz, mz + 1)
    w = torch.exp(-(ky[:, None] ** 2 + kz[None, :] ** 2).double() / 16.0)

    def psi(salt):
        g = _gen(seed, salt)
        a = torch.randn(w.shape, generator=g, dtype=torch.float64)
        b = torch.randn(w.shape, generator=g, dtype=torch.float64)
        c = torch.complex(w * a, -w * b)
        out = []
        for fac in (1.0, 1j * ky[:, None] * (2 * math.pi / (DOMAIN[1][1] - DOMAIN[1][0])),
                    1j * kz[None, :] * (2 * math.pi / (DOMAIN[2][1] - DOMAIN[2][0]))):
            full = torch.zeros(ny, nz, dtype=torch.complex128)
            full[(ky % ny)[:, None], (kz % nz)[None, :]] = c * fac
            out.append((torch.fft.ifft2(full.to(dev)) * (ny * nz)).real)
        return out

    fa, fa_y, _ = psi(1)
    fb, _, fb_z = psi(2)
    u = [env[:, None, None] * (fa_y - fb_z), -denv[:, None, None] * fa, denv[:, None, None] * fb]
    wx = torch.sqrt(1 - x**2) * (math.pi / nx)
    area = (DOMAIN[1][1] - DOMAIN[1][0]) * (DOMAIN[2][1] - DOMAIN[2][0]) / (ny * nz)
    energy = sum((v**2 * wx[:, None, None]).sum() for v in u) * area
    s = torch.sqrt(1e-4 / energy)
    return [(s * v).contiguous() for v in u]


def _spectrum(rows, ny, nz, seed, salt, dev, amplitude=1.0, real=True):
    """Coefficients of a smooth field: decaying in the wall-normal index and in
    |k|, of a real field unless ``real`` is false, Nyquist modes zero."""
    g = _gen(seed, salt)
    shape = (rows, ny, nz)
    f = torch.randn(shape, generator=g, dtype=torch.float64).to(dev)
    if not real:
        f = torch.complex(f, torch.randn(shape, generator=g, dtype=torch.float64).to(dev))
    c = torch.fft.fftn(f, dim=(1, 2)) / math.sqrt(ny * nz)
    ky = torch.fft.fftfreq(ny, 1.0 / ny, dtype=torch.float64, device=dev)
    kz = torch.fft.fftfreq(nz, 1.0 / nz, dtype=torch.float64, device=dev)
    i = torch.arange(rows, dtype=torch.float64, device=dev)
    decay = (1 + i)[:, None, None] ** -3 * torch.exp(
        -(ky[None, :, None] ** 2 + kz[None, None, :] ** 2) / 16.0)
    c = amplitude * decay * c
    c[:, ny // 2, :] = 0
    c[:, :, nz // 2] = 0
    return c.contiguous()


def _member_sizes(case):
    sizes = (case["nx"], case["nx2"], case["nx3"])
    return [sizes[m % 3] for m in range(case["members"])]


def _potential(nx, case, seed, dev):
    return tuple(_spectrum(nx - 2, case["ny"], case["nz"], seed, 10 + k, dev, amplitude=2e-3)
                 for k in range(3))


def _mhd(nx, case, seed, dev):
    """An MHD solver and a developed state of it."""
    solver = PlaneCouetteMHD(N=(nx, case["ny"], case["nz"]), domain=DOMAIN, Re=_re(case),
                             Rm=_re(case), dt=_dt(case), precision=case["precision"])
    flow = solver.state_from_physical(_velocity(nx, case["ny"], case["nz"], "C", seed, dev))
    return solver, MHDState(flow=flow, A=_potential(nx, case, seed, dev))


def _dia(a, dev):
    """The structurally nonzero diagonals of a dense Galerkin matrix."""
    n = a.shape[0]
    offs = [k for k in range(-(n - 1), n) if np.any(np.diagonal(a, k) != 0.0)]
    return DiaMatrix.from_dense(torch.from_numpy(a).to(dev), offsets=offs)


def prepare(case, seed):
    dev = torch.device("cuda")
    kind = case["kind"]
    if kind == "flow":
        n = (case["nx"], case["ny"], case["nz"])
        solver = PlaneCouetteFluctuation(
            N=n, domain=DOMAIN, Re=_re(case), dt=_dt(case), family=case["family"],
            time_integrator=case["integrator"], nonlinear_form=case["form"],
            precision=case["precision"])
        state = solver.state_from_physical(_velocity(*n, case["family"], seed, dev))
        return {"case": case, "solver": solver, "state": solver.solve(state, WARM)}
    if kind == "mhd":
        solver, state = _mhd(case["nx"], case, seed, dev)
        return {"case": case, "solver": solver, "state": solver.solve(state, WARM)}
    if kind == "ensemble":
        pairs = [_mhd(nx, case, 97 * seed + m, dev) for m, nx in enumerate(_member_sizes(case))]
        ens = Ensemble([p[0] for p in pairs])
        return {"case": case, "solver": ens, "state": ens.solve([p[1] for p in pairs], WARM)}
    if kind == "seed":
        n = (case["nx"], case["ny"], case["nz"])
        solver = PlaneCouetteFluctuation(N=n, domain=DOMAIN, Re=_re(case), dt=_dt(case),
                                         time_integrator="SBDF3", nonlinear_form="rotational")
        state = solver.state_from_physical(_velocity(*n, "C", seed, dev))
        return {"case": case, "solver": solver, "state": state}
    if kind == "helmholtz":
        n = (case["nx"], case["ny"])
        solver = Helmholtz2D(n)
        return {"case": case, "solver": solver, "f": _forcing(case, seed, dev)}
    if kind == "transform":
        n = (case["nx"], case["ny"], case["nz"])
        space = TensorProductSpace(case["basis"], n, DOMAIN, padding_factor=(1.0, 1.5, 1.5),
                                   family=case["family"])
        c, u = _transform_inputs(case, seed, dev)
        return {"case": case, "space": space, "c": c, "u": u}
    n = (case["nx"], case["ny"], case["nz"])
    space = TensorProductSpace("D", n, DOMAIN, family=case["family"])
    g0, g2 = space.galerkin(0), space.galerkin(2)
    ky, kz = space.wavenumbers(1), space.wavenumbers(2)

    def diag(v):
        return DiaMatrix(v.reshape(1, -1), [0], (v.numel(), v.numel()))

    one_y, one_z = diag(torch.ones_like(ky)), diag(torch.ones_like(kz))
    op = TPMatrices([TPMatrix([_dia(g2, dev), one_y, one_z], -1.0),
                     TPMatrix([_dia(g0, dev), diag(1.0 + ky**2), one_z]),
                     TPMatrix([_dia(g0, dev), one_y, diag(kz**2)])])
    v, rhs = _kron_inputs(case, seed, dev)
    return {"case": case, "op": op, "solver": tpmats_wavenumber_factor(op), "v": v, "rhs": rhs}


def _forcing(case, seed, dev):
    """Orthogonal Chebyshev x Fourier coefficients of a smooth real forcing."""
    c = _spectrum(case["nx"], case["ny"], 4, seed, 20, dev)[:, :, 0]
    j = torch.arange(case["ny"], device=dev)
    return (0.5 * (c + torch.conj(c[:, (-j) % case["ny"]]))).contiguous()


def _transform_inputs(case, seed, dev):
    rows = case["nx"] - {"C": 0, "D": 2, "B": 4}[case["basis"]]
    m = [max(n, int(1.5 * n)) if case["padded"] else n for n in (case["ny"], case["nz"])]
    c = _spectrum(rows, case["ny"], case["nz"], seed, 30, dev)
    g = _gen(seed, 31)
    u = torch.randn((case["nx"], *m), generator=g, dtype=torch.float64).to(dev)
    return c, u.to(torch.complex128)


def _kron_inputs(case, seed, dev):
    shape = (case["nx"] - 2, case["ny"], case["nz"])
    v = _spectrum(*shape, seed, 40, dev)
    rhs = torch.stack([_spectrum(*shape, seed, 41 + r, dev) for r in range(case["rhs"])])
    return v, rhs


# -- one pass ------------------------------------------------------------------


def _flow_outputs(st: KMMState):
    return {"u": st.u, "g": st.g, "nonlinear_old": st.nonlinear_old,
            "nonlinear_older": st.nonlinear_older, "solution_old": st.solution_old,
            "solution_older": st.solution_older}


def _mhd_outputs(st: MHDState):
    return {"flow": _flow_outputs(st.flow), "A": st.A, "nonlinear_A_old": st.nonlinear_A_old,
            "nonlinear_A_older": st.nonlinear_A_older, "A_old": st.A_old,
            "A_older": st.A_older}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("flow", "mhd"):
        solver = state["solver"]
        if case["steps"] == 1:
            st = solver.step(state["state"])
        else:
            st = solver.solve(state["state"], case["steps"])
        out = _flow_outputs(st) if kind == "flow" else _mhd_outputs(st)
        return {"state": out, "diagnostics": solver.diagnostics_tensor(st)}
    if kind == "ensemble":
        sts = state["solver"].solve(state["state"], case["steps"])
        # the evolved fields of every member (their histories would be 35 arrays each)
        return [{"u": st.flow.u, "g": st.flow.g, "A": st.A} for st in sts]
    if kind == "seed":
        gain, grad = gain_and_gradient(state["solver"], state["state"], case["steps"],
                                       checkpoint=case["checkpoint"])
        return {"gain": gain, "u": grad.u, "g": grad.g}
    if kind == "helmholtz":
        return state["solver"](state["f"])
    if kind == "transform":
        space, pad = state["space"], case["padded"]
        return {"u": space.backward(state["c"], padded=pad),
                "dudx": space.backward_primitive(state["c"], (1, 0, 0), padded=pad),
                "c": space.forward(state["u"], padded=pad)}
    return {"Av": state["op"] @ state["v"], "x": state["solver"].solve_many(state["rhs"])}


# -- what a pass cannot do without ------------------------------------------------


def _fft_flops(n):
    return 5.0 * n * math.log2(n)


def _transform_flops(nx, ny, nz, fields):
    """Half-spectrum y and z transforms of ``fields`` fields on the 3/2 grid
    and a fast x transform of each."""
    my, mz = int(1.5 * ny), int(1.5 * nz)
    return fields * (nx * (nz // 2) * _fft_flops(my) + nx * my * 0.5 * _fft_flops(mz)
                     + ny * (nz // 2) * 2 * _fft_flops(nx))


def work(case):
    kind = case["kind"]
    if kind == "helmholtz":
        n, m = case["nx"], case["ny"]
        return {"bytes": 2 * 16 * n * m,
                "flops": 3 * m * 4.0 * n * n + 3 * n * _fft_flops(m) + m * 4.0 * n * n}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    e = nx * ny * nz
    if kind == "transform":
        my, mz = (int(1.5 * ny), int(1.5 * nz)) if case["padded"] else (ny, nz)
        phys = nx * my * mz
        one = nx * nz * _fft_flops(my) + nx * my * _fft_flops(mz)
        return {"bytes": 16 * (3 * phys + 3 * e), "flops": 3 * (one + 4.0 * nx * e)}
    if kind == "kron":
        bands = 4 if case["family"] == "L" else 1 + nx // 2
        return {"bytes": 16 * e * (2 + 2 * case["rhs"]) + 8 * e * bands / 2,
                "flops": 4.0 * e * bands * (1 + case["rhs"])}
    members = [nx]
    if kind == "ensemble":
        members = _member_sizes(case)
    mhd = kind in ("mhd", "ensemble")
    total = {"bytes": 0.0, "flops": 0.0}
    for n in members:
        es = 16 * n * ny * nz  # one full complex field
        levels = 14 if mhd else 8  # state fields read / written by set and get
        stages = {"IMEXRK222": 2, "IMEXRK3": 3}.get(case.get("integrator"), 1)
        # per step: two evolved fields (five with A), three levels and two
        # nonlinear levels read, one of each written, half spectra
        per_step = (5 + 2) * (5 if mhd else 2) * es / 2
        fields = 18 if mhd else 12 if case.get("form") == "gradient" else 9
        flops = stages * _transform_flops(n, ny, nz, fields)
        steps = case["steps"] * (3 if kind == "seed" else 1)
        total["bytes"] += 2 * levels * es + steps * stages * per_step
        total["flops"] += steps * flops
    return total


# -- the same in plain torch, 64 bits -----------------------------------------------


class _X:
    """Wall-normal axis: Vandermonde matrix, derivative, stencils, mass."""

    def __init__(self, family, n, dev):
        poly = np.polynomial.legendre if family == "L" else np.polynomial.chebyshev
        x = _nodes(family, n)
        v = (poly.legvander if family == "L" else poly.chebvander)(x, n - 1)
        k = np.arange(n)
        if family == "L":
            w, norms = poly.leggauss(n)[1], 2.0 / (2 * k + 1.0)
            s2, s4 = 2 * (-2 * k - 5) / (2 * k + 7), (2 * k + 3) / (2 * k + 7)
        else:
            w, norms = np.full(n, np.pi / n), np.where(k == 0, np.pi, np.pi / 2)
            s2, s4 = 2 * (-k - 2.0) / (k + 3), (k + 1.0) / (k + 3)
        der = poly.legder if family == "L" else poly.chebder
        d = np.zeros((n, n))
        d[: n - 1] = der(np.eye(n), axis=0)
        integ = np.zeros(n)
        integ[::2] = [2.0 if (family == "L" and j == 0) else 0.0 if family == "L"
                      else 2.0 / (1 - j * j) for j in k[::2]]
        stencil = {"C": np.eye(n), "D": np.zeros((n - 2, n)), "B": np.zeros((n - 4, n))}
        for i in range(n - 2):
            stencil["D"][i, [i, i + 2]] = 1.0, -1.0
        for i in range(n - 4):
            stencil["B"][i, [i, i + 2, i + 4]] = 1.0, s2[i], s4[i]
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(dev)  # noqa: E731
        self.x, self.V, self.Q, self.D, self.W = t(x), t(v), t(v.T * w), t(d), t(norms)
        self.S = {b: t(s) for b, s in stencil.items()}
        self.fejer = torch.linalg.solve(self.V.T, t(integ))  # weights of the plain integral

    def gal(self, b, k):
        """(phi_i, d^k phi_j)_w"""
        return (self.S[b] * self.W) @ torch.linalg.matrix_power(self.D, k) @ self.S[b].T

    def project(self, b, orth):
        """Galerkin projection of orthogonal coefficients."""
        return _mul(torch.linalg.solve(self.gal(b, 0), self.S[b] * self.W), orth)

    def forward(self, b, samples):
        return _mul(torch.linalg.solve(self.gal(b, 0), self.S[b] @ self.Q), samples)


def _mul(a, c):
    """Real matrix along the first axis of a (complex) array."""
    if not c.is_complex():
        return torch.tensordot(a, c, dims=1)
    return torch.complex(torch.tensordot(a, c.real, dims=1), torch.tensordot(a, c.imag, dims=1))


class _Periodic:
    def __init__(self, ny, nz, dev, pad=1.5):
        self.n, self.m = (ny, nz), (max(ny, int(pad * ny)), max(nz, int(pad * nz)))
        f = lambda n: torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=dev)  # noqa: E731
        iy, iz = f(ny), f(nz)
        ly, lz = (d[1] - d[0] for d in DOMAIN[1:])
        self.ky = (iy * (2 * math.pi / ly))[None, :, None]
        self.kz = (iz * (2 * math.pi / lz))[None, None, :]
        self.k2 = self.ky**2 + self.kz**2
        self.mask = ((iy != -ny // 2)[None, :, None] & (iz != -nz // 2)[None, None, :]).double()
        self.jy, self.jz = iy.long() % self.m[0], iz.long() % self.m[1]
        self.area, self.weight = ly * lz, ly * lz

    def backward(self, c, padded=True):
        if not padded or self.m == self.n:
            return torch.fft.ifft2(c) * (self.n[0] * self.n[1])
        full = torch.zeros((c.shape[0], *self.m), dtype=c.dtype, device=c.device)
        full = full.index_put((torch.arange(c.shape[0], device=c.device)[:, None, None],
                               self.jy[None, :, None], self.jz[None, None, :]), c)
        return torch.fft.ifft2(full) * (self.m[0] * self.m[1])

    def forward(self, u):
        c = torch.fft.fft2(u) / (u.shape[1] * u.shape[2])
        if tuple(u.shape[1:]) == self.n:
            return c
        return c[:, self.jy][:, :, self.jz]


_A3, _B3 = (8 / 15, 5 / 12, 3 / 4), (0.0, -17 / 60, -5 / 12)
_G2 = (2 - math.sqrt(2)) / 2
_D2 = 1 - 1 / (2 * _G2)


class _Couette:
    """Velocity-vorticity Couette flow, optionally with a vector potential."""

    def __init__(self, case, nx, mhd, dev):
        self.x = x = _X(case.get("family", "C"), nx, dev)
        self.p = p = _Periodic(case["ny"], case["nz"], dev)
        self.dt, self.nu, self.mhd = _dt(case), 1 / _re(case), mhd
        self.grad = case.get("form") == "gradient"
        self.kind = case.get("integrator", "SBDF3")
        self.g = {b: [x.gal(b, k) for k in (0, 2, 4)] for b in "BD"}
        self.mean = torch.zeros_like(p.k2)
        self.mean[0, 0, 0] = 1.0
        self.inv_k2 = torch.where(p.k2 == 0, 0.0, 1 / torch.where(p.k2 == 0, 1.0, p.k2))
        self.proj = torch.linalg.solve(x.gal("D", 0), x.S["D"] * x.W)
        self.factors = {}

    # linear operators of the evolved fields (u0, g, v00, w00[, A]); M + c L
    def rows(self, s, c):
        p, w = self.p, self.p.weight

        def lap(b, f, coef):
            x0, x2 = _mul(self.g[b][0], f), _mul(self.g[b][1], f)
            return w * (x0 + coef * (x2 - p.k2 * x0))

        u = s[0]
        x0, x2, x4 = (_mul(m, u) for m in self.g["B"])
        out = [w * (x2 - p.k2 * x0 + c * self.nu * (x4 - 2 * p.k2 * x2 + p.k2**2 * x0)),
               lap("D", s[1], c * self.nu)]
        m00 = self.g["D"][0] + c * self.nu * self.g["D"][1]
        out += [m00 @ s[2], m00 @ s[3]]
        return out + [lap("D", a, c * self.nu) for a in s[4:]]

    def solve(self, gamma, r):
        """(M - gamma L) x = r, the Nyquist modes masked."""
        if gamma not in self.factors:
            p, gn = self.p, gamma * self.nu
            ny, nz = p.n
            k2 = p.k2[0, : ny // 2 + 1, : nz // 2 + 1, None, None]
            b0, b2, b4 = self.g["B"]
            d0, d2, _ = self.g["D"]
            su = b2 - k2 * b0 - gn * (b4 - 2 * k2 * b2 + k2**2 * b0)
            sg = d0 - gn * (d2 - k2 * d0)
            iy = torch.minimum(torch.arange(ny), ny - torch.arange(ny)).to(k2.device)
            iz = torch.minimum(torch.arange(nz), nz - torch.arange(nz)).to(k2.device)
            full = [torch.linalg.inv(m)[iy][:, iz] / p.weight for m in (su, sg)]
            self.factors[gamma] = (*full, torch.linalg.inv(d0 - gn * d2))
        su, sg, s00 = self.factors[gamma]

        def apply(m, c):
            v = torch.view_as_real(c * self.p.mask).permute(1, 2, 0, 3)
            return torch.view_as_complex((m @ v).contiguous()).permute(2, 0, 1) * self.p.mask

        return [apply(su, r[0]), apply(sg, r[1]), s00 @ r[2], s00 @ r[3],
                *(apply(sg, a) for a in r[4:])]

    def velocity(self, s):
        """(u0, u1, u2) of the evolved fields."""
        p = self.p
        f = _mul(self.proj @ self.x.D @ self.x.S["B"].T, s[0])
        u1 = 1j * self.inv_k2 * (p.ky * f + p.kz * s[1])
        u2 = 1j * self.inv_k2 * (p.kz * f - p.ky * s[1])
        return [s[0], p.mask * u1 + self.mean * s[2][:, None, None],
                p.mask * u2 + self.mean * s[3][:, None, None]]

    def phys(self, orth):
        return self.p.backward(_mul(self.x.V, orth * self.p.mask)).real

    def forward(self, b, u):
        return self.x.forward(b, self.p.forward(u.to(torch.complex128)) * self.p.mask)

    def nonlinear(self, u, a=()):
        """Nonlinear rows of (u0, g, v00, w00[, A])."""
        x, p = self.x, self.p
        uo = [_mul(x.S[b].T, c) for b, c in zip("BDD", u)]
        dx = [_mul(x.D, c) for c in uo]
        up, xb = [self.phys(c) for c in uo], x.x[:, None, None]
        iy, iz = 1j * p.ky, 1j * p.kz
        if self.grad:
            n = [sum(q * self.phys(t) for q, t in zip(up, (dx[i], iy * uo[i], iz * uo[i])))
                 + xb * self.phys(iy * uo[i]) for i in range(3)]
            n[1] = n[1] + up[0]
        else:
            om = [self.phys(iy * uo[2] - iz * uo[1]), self.phys(iz * uo[0] - dx[2]),
                  self.phys(dx[1] - iy * uo[0]) + 1.0]
            n = [-c for c in _cross([up[0], up[1] + xb, up[2]], om)]
        extra = []
        if self.mhd:
            ao = [_mul(x.S["D"].T, c) for c in a]
            b = [iy * ao[2] - iz * ao[1], iz * ao[0] - _mul(x.D, ao[2]),
                 _mul(x.D, ao[1]) - iy * ao[0]]
            td = lambda c: _mul(x.S["D"].T, _mul(self.proj, c))  # noqa: E731
            j = [iy * b[2] - iz * b[1], td(iz * b[0] - _mul(x.D, b[2])),
                 td(_mul(x.D, b[1]) - iy * b[0])]
            bp, jp = [self.phys(c) for c in b], [self.phys(c) for c in j]
            n = [c - e for c, e in zip(n, _cross(jp, bp))]
            emf = _cross([up[0], up[1] + xb, up[2]], bp)
            extra = [p.weight * _mul(self.g["D"][0], self.forward("D", c)) for c in emf]
        h = [self.forward("D", c) for c in n]
        ho = [_mul(x.S["D"].T, c) for c in h]
        hu = _mul(x.D, iy * ho[1] + iz * ho[2]) + p.k2 * ho[0]
        hg = iz * ho[1] - iy * ho[2]
        rows = [p.weight * _mul(x.S["B"] * x.W, hu), p.weight * _mul(x.S["D"] * x.W, hg)]
        means = [-(self.g["D"][0] @ c[:, 0, 0].real) for c in h[1:]]
        return [*rows, *means, *extra]

    def evolved(self, u, g, a=()):
        return [u[0], g, u[1][:, 0, 0].real, u[2][:, 0, 0].real, *a]

    def start(self, fields):
        u = [self.forward(b, f) for b, f in zip("BDD", fields)]
        return u, 1j * self.p.ky * u[2] - 1j * self.p.kz * u[1]

    def rollout(self, u, g, a, steps):
        """``steps`` steps from a state without history: (u, evolved fields,
        previous evolved levels, previous nonlinear levels)."""
        s, old_s, old_n = self.evolved(u, g, a), [], []
        for n in range(steps):
            cur = self.nonlinear(u, a)
            if self.kind == "IMEXRK222":
                s1 = self.solve(_G2 * self.dt, _comb((1, self.rows(s, 0.0)), (_G2 * self.dt, cur)))
                n1 = self.nonlinear(self.velocity(s1))
                lin = _comb((1, self.rows(s1, 1.0)), (-1, self.rows(s1, 0.0)))
                new = self.solve(_G2 * self.dt, _comb(
                    (1, self.rows(s, 0.0)), (_D2 * self.dt, cur), ((1 - _D2) * self.dt, n1),
                    ((1 - _G2) * self.dt, lin)))
            elif self.kind == "CNAB2":
                terms = [(1, self.rows(s, 0.5 * self.dt)),
                         ((1.5 if old_n else 1.0) * self.dt, cur)]
                terms += [(-0.5 * self.dt, old_n[0])] if old_n else []
                new = self.solve(0.5 * self.dt, _comb(*terms))
            elif self.kind == "IMEXRK3" or n < 2:
                st, prev, now = s, None, cur
                for k in range(3):
                    gamma = (_A3[k] + _B3[k]) * self.dt / 2
                    if k:
                        now = self.nonlinear(self.velocity(st), st[4:])
                    terms = [(1, self.rows(st, gamma)), (_A3[k] * self.dt, now)]
                    terms += [(_B3[k] * self.dt, prev)] if k else []
                    st, prev = self.solve(gamma, _comb(*terms)), now
                new = st
            else:
                c = 1 / 11
                lv = _comb((18 * c, s), (-9 * c, old_s[0]), (2 * c, old_s[1]))
                new = self.solve(6 / 11 * self.dt, _comb(
                    (1, self.rows(lv, 0.0)), (18 * c * self.dt, cur),
                    (-18 * c * self.dt, old_n[0]), (6 * c * self.dt, old_n[1])))
            old_s, old_n = [s, *old_s][:2], [cur, *old_n][:2]
            s, a = new, new[4:]
            u = self.velocity(s)
        return u, s, old_s, old_n

    def energy(self, u):
        """(sum_f int |u_f|^2 and the samples of u on the unpadded mesh)"""
        up = [self.p.backward(_mul(self.x.V @ self.x.S[b].T, c), False).real
              for b, c in zip("BDD", u)]
        w = self.x.fejer[:, None, None] * (self.p.area / (self.p.n[0] * self.p.n[1]))
        return sum((w * v**2).sum() for v in up), up, w

    def diagnostics(self, u):
        ep, up, w = self.energy(u)
        xb = self.x.x[:, None, None]
        et = ep + (w * (2 * up[1] * xb + xb**2)).sum()
        x = self.x
        orth = [_mul(x.S[b].T, c) for b, c in zip("BDD", u)]
        div = self.p.backward(_mul(x.V, _mul(x.D, orth[0]) + 1j * self.p.ky * orth[1]
                                   + 1j * self.p.kz * orth[2]), False)
        m = orth[1][:, 0, 0].real
        k = torch.arange(m.numel(), dtype=torch.float64, device=m.device)
        sign = 1 - 2 * (k % 2)
        dm = x.D @ m
        return torch.stack([ep, et, torch.sqrt((w * div.abs() ** 2).sum()), m.sum() + 1.0,
                            (sign * m).sum() - 1.0, dm.sum() + 1.0, (sign * dm).sum() + 1.0,
                            0.5 * (x.fejer * (x.V @ dm)).sum() + 1.0])


def _cross(a, b):
    return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]


def _comb(*terms):
    return [sum(c * f for c, f in zip([t[0] for t in terms], fs))
            for fs in zip(*(t[1] for t in terms))]


def _exact_flow(case, nx, seed, mhd, dev):
    m = _Couette(case, nx, mhd, dev)
    u, g = m.start(_velocity(nx, case["ny"], case["nz"], case.get("family", "C"), seed, dev))
    a = _potential(nx, case, seed, dev) if mhd else ()
    u, s, old_s, old_n = m.rollout(u, g, a, WARM + case["steps"])
    out = {"u": u, "g": s[1]}
    if m.kind == "SBDF3":
        out |= {"nonlinear_old": old_n[0][:4], "nonlinear_older": old_n[1][:4],
                "solution_old": old_s[0][:4], "solution_older": old_s[1][:4]}
    elif m.kind == "CNAB2":
        out["nonlinear_old"] = old_n[0]
    if not mhd:
        return {"state": out, "diagnostics": m.diagnostics(u)}
    state = {"flow": out, "A": s[4:], "nonlinear_A_old": old_n[0][4:],
             "nonlinear_A_older": old_n[1][4:], "A_old": old_s[0][4:], "A_older": old_s[1][4:]}
    return {"state": state, "diagnostics": None}


def exact(case, seed):
    dev = _device()
    kind = case["kind"]
    if kind in ("flow", "mhd"):
        return _exact_flow(case, case["nx"], seed, kind == "mhd", dev)
    if kind == "ensemble":
        outs = [_exact_flow(case, nx, 97 * seed + m, True, dev)["state"]
                for m, nx in enumerate(_member_sizes(case))]
        return [{"u": o["flow"]["u"], "g": o["flow"]["g"], "A": o["A"]} for o in outs]
    if kind == "seed":
        m = _Couette(case, case["nx"], False, dev)
        u, g = m.start(_velocity(case["nx"], case["ny"], case["nz"], "C", seed, dev))
        leaves = [t.detach().requires_grad_() for t in (*u, g)]
        end = m.rollout(leaves[:3], leaves[3], (), case["steps"])[0]
        gain = m.energy(end)[0] / m.energy(leaves[:3])[0]
        gr = [torch.conj(t).resolve_conj() for t in torch.autograd.grad(gain, leaves)]
        return {"gain": float(gain.detach()), "u": gr[:3], "g": gr[3]}
    if kind == "helmholtz":
        x = _X("C", case["nx"], dev)
        f = _mul(x.V, _forcing(case, seed, dev))
        k = torch.fft.fftfreq(case["ny"], 1.0 / case["ny"], dtype=torch.float64, device=dev)
        a = -x.gal("D", 2) + (1.0 + k[:, None, None] ** 2) * x.gal("D", 0)
        rhs = _mul(x.S["D"] @ x.Q, f)
        sol = torch.linalg.solve(a.to(torch.complex128), rhs.T[:, :, None])[:, :, 0].T
        return torch.fft.ifft(_mul(x.V @ x.S["D"].T, sol), dim=1) * case["ny"]
    x = _X(case["family"], case["nx"], dev)
    p = _Periodic(case["ny"], case["nz"], dev, 1.5 if case.get("padded") else 1.0)
    if kind == "transform":
        c, u = _transform_inputs(case, seed, dev)
        orth = _mul(x.S[case["basis"]].T, c)
        return {"u": p.backward(_mul(x.V, orth)), "dudx": p.backward(_mul(x.V @ x.D, orth)),
                "c": x.forward(case["basis"], p.forward(u))}
    v, rhs = _kron_inputs(case, seed, dev)
    g0, g2 = x.gal("D", 0), x.gal("D", 2)
    av = -_mul(g2, v) + (1.0 + p.k2) * _mul(g0, v)
    a = -g2 + (1.0 + p.k2[0, :, :, None, None]) * g0
    r = torch.view_as_real(rhs).permute(2, 3, 1, 0, 4).flatten(3)
    sol = torch.linalg.solve(a, r).unflatten(3, (case["rhs"], 2)).permute(3, 2, 0, 1, 4)
    return {"Av": av, "x": torch.view_as_complex(sol.contiguous())}
