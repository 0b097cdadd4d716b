"""The engine's work as its users run it: one timed case per way of calling it.

A case is a dict of plain values. ``prepare`` makes what a program holds before the call (a grid with
its potential, device states, field samples), ``run`` is one pass through the public entry points, and
``exact`` is the same result from plain torch in 64 bits.

    kind       the entry point of a pass
    imag       Grid.imag_propagate for every state, then Grid.energies (an eigenstate job)
    length     Grid.run_length with observables at every step (a length-gauge propagation)
    velocity   Grid.run_velocity with observables at every step
    step       Grid.integration_step_length of one step (a driver that steps by itself)
    sweep      batch.launch over members of several grid sizes
    adjoint    adjoint.length_gauge_objective and its backward
    spectra    Grid.observables (k-space ones among them) and Grid.final_spectra of a final state

Propagations go on from where the last pass left the state, as a program's loop does.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from tdse_nd_mpi_b200 import Grid
from tdse_nd_mpi_b200.adjoint import length_gauge_objective
from tdse_nd_mpi_b200.batch import Member, launch
from tdse_nd_mpi_b200.batch import prepare as prepare_members

DT = 0.05
W800 = 45.5637639947958 / 800.0  # angular frequency of 800 nm light in atomic units


def listed():
    return [
        # one time step of a small 2-D grid per call: a driver that writes its own loop
        {"name": "step_2d_128", "kind": "step", "shape": "128x128", "dr": 0.2, "integrator": "BM4",
         "precision": "fp64", "steps": 1, "potential": "H_2D"},
        # a 1-D model atom in a laser field, the drivers' everyday size
        {"name": "h1d_real_512", "kind": "length", "shape": "512", "dr": 0.2, "integrator": "BM4",
         "precision": "fp64", "steps": 32, "potential": "H_1D", "obs": "norm,dipole_r"},
        # the H_1D eigenstate job: four states in imaginary time with Gram-Schmidt at every step
        {"name": "h1d_imag_4096", "kind": "imag", "shape": "4096", "dr": 0.1, "integrator": "BM4",
         "precision": "fp64", "steps": 48, "potential": "H_1D", "states": 4},
        # a long 1-D box (the drivers' example size): ionised electrons stay on the grid
        {"name": "h1d_real_262144", "kind": "length", "shape": "262144", "dr": 0.1, "integrator": "BM4",
         "precision": "fp64", "steps": 16, "potential": "H_1D", "obs": "norm,dipole_r"},
        # the benchmark's workload: absorbing mask as a CAP, norm, dipole and acceleration every step
        {"name": "h2d_real_1024", "kind": "length", "shape": "1024x1024", "dr": 0.2, "integrator": "BM4",
         "precision": "fp64", "steps": 48, "potential": "soft", "obs": "norm,dipole_r,accel"},
        # the same in mixed precision
        {"name": "h2d_real_1024_mixed", "kind": "length", "shape": "1024x1024", "dr": 0.2, "integrator": "BM4",
         "precision": "mixed", "steps": 48, "potential": "soft", "obs": "norm,dipole_r,accel"},
        # the Ne_2D-style job's two halves: eigenstates in mixed precision, then the field run in FP64
        {"name": "ne2d_imag_2048_mixed", "kind": "imag", "shape": "2048x2048", "dr": 0.15, "integrator": "BM6",
         "precision": "mixed", "steps": 6, "potential": "Ne_2D", "states": 3},
        {"name": "ne2d_real_2048", "kind": "length", "shape": "2048x2048", "dr": 0.15, "integrator": "BM6",
         "precision": "fp64", "steps": 8, "potential": "Ne_2D", "obs": "norm,dipole_r"},
        # velocity gauge on an elongated 3-D box
        {"name": "h3d_velocity_64_256_128", "kind": "velocity", "shape": "64x256x128", "dr": 0.3,
         "integrator": "RKN4", "precision": "fp64", "steps": 8, "potential": "soft", "obs": "norm,dipole_r"},
        # gradient of the absorbed norm with respect to the field samples
        {"name": "h3d_adjoint_128", "kind": "adjoint", "shape": "128x128x128", "dr": 0.3, "integrator": "BM4",
         "precision": "fp64", "steps": 10, "potential": "soft", "checkpoint": 5, "radius": 3.0},
        # a sweep over CEP and intensity on uneven grids, mixed precision, BM4 and Verlet members
        {"name": "sweep_mixed", "kind": "sweep", "n256": 6, "n512": 9, "n1024": 3, "dr": 0.2,
         "precision": "mixed", "steps": 16, "potential": "H_2D", "obs": "norm,dipole_r"},
        # the analysis at the end of a run: k-space observables, photoelectron spectra
        {"name": "spectra_2d_512", "kind": "spectra", "shape": "512x512", "dr": 0.2, "integrator": "BM4",
         "precision": "fp64", "steps": 1, "potential": "H_2D", "obs": "norm,dipole_r,dipole_v,energy,Lz",
         "ne": 400, "de": 0.01, "prmax": 2.0},
    ]


def draw(rng):
    """One more case of the listed kinds and size ranges: grids of 1 to 3 dimensions with axes of
    different lengths, every integrator, both precisions."""
    kind = rng.choice(["imag", "length", "length", "length", "velocity", "step", "adjoint", "sweep", "spectra"])
    c = {"kind": kind, "dr": round(rng.uniform(0.1, 0.3), 3), "integrator": rng.choice(["Verlet", "BM4", "BM6", "RKN4"]),
         "precision": rng.choice(["fp64", "fp64", "mixed"])}
    if kind == "sweep":
        c |= {"n256": rng.randint(1, 8), "n512": rng.randint(0, 8), "n1024": rng.randint(0, 3), "precision": "mixed",
              "steps": rng.randint(8, 24), "potential": "H_2D", "obs": "norm,dipole_r"}
        return c
    dim = rng.choice([1, 1, 2, 2, 2, 3]) if kind not in ("adjoint", "spectra") else rng.choice([2, 3] if kind == "adjoint" else [1, 2])
    if dim == 1:
        logs = [rng.randint(8, 18 if kind in ("length", "imag") else 12)]
    else:
        top = {"adjoint": 21, "spectra": 18, "step": 20}.get(kind, 22)
        while True:  # axes of their own lengths, not one more size of a square
            logs = [rng.randint(5, 12 if dim == 2 else 9) for _ in range(dim)]
            if 12 <= sum(logs) <= top:
                break
    work = {"adjoint": 1 << 23, "spectra": 1 << 18, "step": 1}.get(kind, 1 << 25)
    steps = max(2, min(rng.randint(6, 48), work >> sum(logs)))
    if kind == "adjoint":
        steps, c["precision"] = min(steps, 12), "fp64"
    if kind == "spectra":
        c["precision"] = "fp64"
    c |= {"shape": "x".join(str(1 << k) for k in logs), "steps": 1 if kind in ("step", "spectra") else steps,
          "potential": "soft" if dim == 3 or rng.random() < 0.5 else ("H_1D" if dim == 1 else rng.choice(["H_2D", "Ne_2D"]))}
    if kind == "imag":
        c["states"] = rng.randint(1, 4)
    if kind in ("length", "velocity"):
        c["obs"] = rng.choice(["norm", "norm,dipole_r", "dipole_r,norm"] + (["norm,dipole_r,accel"] if c["potential"] == "soft" else []))
    if kind == "adjoint":
        c |= {"checkpoint": rng.randint(1, 8), "radius": round(rng.uniform(1.5, 4.0), 2)}
    if kind == "spectra":
        c |= {"obs": "norm,dipole_r,dipole_v,energy,Lz", "ne": rng.randint(50, 400), "de": 0.01,
              "prmax": round(rng.uniform(1.0, 3.0), 2)}
    return c


# ---------------------------------------------------------------- inputs


def _shape(case):
    return tuple(int(v) for v in case["shape"].split("x"))


def _axes(shape, dr):
    return [-0.5 * dr * n + dr * torch.arange(n, dtype=torch.float64, device="cuda") for n in shape]


def _spread(ax, j, dim):
    return ax.reshape([-1 if k == j else 1 for k in range(dim)])


def _radius2(shape, dr):
    return sum(_spread(a, j, len(shape)) ** 2 for j, a in enumerate(_axes(shape, dr)))


def _potential(case, shape):
    """V on the grid (the named potentials are those of the parameter files)."""
    r2 = _radius2(shape, case["dr"])
    name = case["potential"]
    if name == "H_1D":
        return -1.0 / torch.sqrt(r2 + 2.0)
    if name == "H_2D":
        return -1.0 / torch.sqrt(r2 + 0.7396)
    if name == "Ne_2D":
        return -(1.0 + 9.0 * torch.exp(-r2)) / torch.sqrt(r2 + 2.88172)
    return -1.0 / torch.sqrt(r2 + 0.64)


def _cap_axis(n, dr):
    """The absorber along one axis: -log of a cos^(1/8) mask over the outer 10%, per unit of time."""
    x = np.abs(-0.5 * dr * n + np.arange(n) * dr)
    half, edge = 0.5 * dr * n, 0.45 * dr * n
    mask = np.ones(n)
    out = x > edge
    mask[out] = np.cos(0.5 * np.pi * (x[out] - edge) / (half - edge)).clip(0.0) ** 0.125
    return -np.log(np.maximum(mask, 8e-3)) / DT


def _vcap(shape, dr):
    caps = [torch.from_numpy(_cap_axis(n, dr)).cuda() for n in shape]
    return sum(_spread(v, j, len(shape)) for j, v in enumerate(caps)).expand(shape).contiguous()


def _packet(shape, dr, gen, noise=0.0):
    """A bound-state-like packet with a seeded momentum, normalised; noise: the share of white noise
    in it (the imaginary-time guesses)."""
    k = (torch.rand(len(shape), generator=gen, dtype=torch.float64, device="cuda") - 0.5) * 1.5
    phase = sum(_spread(a, j, len(shape)) * k[j] for j, a in enumerate(_axes(shape, dr)))
    psi = torch.exp(-0.5 * _radius2(shape, dr)) * torch.exp(1j * phase)
    if noise:
        psi = psi + noise * torch.randn(shape, generator=gen, dtype=torch.complex128, device="cuda")
    return psi / torch.sqrt((psi.abs() ** 2).sum() * dr ** len(shape))


COEFFICIENTS = {
    "Verlet": [.5],
    "BM4": [.0792036964311957, .1303114101821663, .2228614958676077, -.3667132690474257, .3246481886897062,
            .1096884778767498],
    "BM6": [.050262764400392, .098553683500650, .314960616927694, -.447346482695478, .492426372489876,
            -.425118767797691, .237063913978122, .195602488600053, .346358189850727, -.362762779254345],
    "RKN4": [.082984406417405, .162314550766866, .233995250731502, .370877414979578, -.409933719901926,
             .059762097006575],
}


def _as(integrator):
    a = COEFFICIENTS[integrator]
    return [v * DT for v in a + a[::-1]]


def _field(steps, s, dim, gen):
    """Samples of an 800 nm pulse near its maximum: intensity and carrier phase from the seed, nearly
    linear along the first axis."""
    u = torch.rand(2, generator=gen, dtype=torch.float64, device="cuda").cpu().numpy()
    f0 = 5.33803e-9 * math.sqrt(5e13 * 6.0 ** u[0])
    t = (np.arange(steps)[:, None] + (np.arange(s) + 0.5) / s) * DT
    F = np.zeros((steps, s, dim))
    F[:, :, 0] = f0 * np.sin(W800 * t + 2 * np.pi * u[1])
    if dim > 1:
        F[:, :, 1] = 0.1 * f0 * np.cos(W800 * t + 2 * np.pi * u[1])
    return F


def _inputs(case, seed):
    """Everything seeded, on the GPU: shared by prepare and exact."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    shape = _shape(case)
    s = len(COEFFICIENTS[case["integrator"]])
    d = {"shape": shape, "dim": len(shape), "s": s}
    kind = case["kind"]
    if kind == "imag":
        d["psi"] = [_packet(shape, case["dr"], gen, 0.05) for _ in range(case["states"])]
    else:
        d["psi"] = _packet(shape, case["dr"], gen, 0.01 if kind == "spectra" else 0.0)
    if kind == "step":  # in the momentum representation, where that entry point takes it
        d["psi"] = torch.fft.fftn(d["psi"]) / math.sqrt(d["psi"].numel())
    if kind in ("length", "velocity", "step", "adjoint"):
        d["field"] = _field(case["steps"], s, len(shape), gen)
    if kind == "velocity":
        d["field"] = d["field"] / W800
        d["alpha"] = np.ascontiguousarray(d["field"][:, 0, :])
    if kind == "spectra":
        d["alpha"] = _field(1, 1, len(shape), gen)[0, 0] / W800
    return d


def _members(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    out = []
    for k, n in enumerate([256] * case["n256"] + [512] * case["n512"] + [1024] * case["n1024"]):
        integ = "BM4" if k % 2 == 0 else "Verlet"
        out.append(({"shape": f"{n}x{n}", "dr": case["dr"], "integrator": integ, "potential": case["potential"],
                     "steps": case["steps"], "obs": case["obs"]},
                    _packet((n, n), case["dr"], gen), _field(case["steps"], len(COEFFICIENTS[integ]), 2, gen)))
    return out


def _device_state(psi, precision):
    return psi.to(torch.complex128 if precision == "fp64" else torch.complex64).contiguous()


def prepare(case, seed):
    if case["kind"] == "sweep":
        runs = []
        for m, psi, E in _members(case, seed):
            member = Member(shape=_shape(m), dr=(m["dr"],) * 2, integrator=m["integrator"], dt=DT,
                            potential=m["potential"], field=E, psi0=psi.cpu().numpy(), cap=(0.05, 5.0),
                            names=tuple(m["obs"].split(",")), precision=case["precision"])
            g, _, E_dev, obs, nv, names = prepare_members([member])[0]
            runs.append((g, _device_state(psi, case["precision"]), E_dev, obs, nv, names))
        return {"case": case, "runs": runs}
    d = _inputs(case, seed)
    shape, dim = d["shape"], d["dim"]
    g = Grid(dim, shape, (case["dr"],) * dim, case["integrator"], DT, precision=case["precision"])
    V = _potential(case, shape)
    if case["potential"] == "soft":
        g.set_potential(V.cpu().numpy())
        r2 = _radius2(shape, case["dr"])
        for j, a in enumerate(_axes(shape, case["dr"])):
            if "accel" in case.get("obs", ""):
                g.set_gradv(j, (_spread(a, j, dim) / (r2 + 0.64) ** 1.5).cpu().numpy())
    else:
        g.set_potential(case["potential"])
    if case["kind"] not in ("imag", "spectra"):
        g.set_vcap(_vcap(shape, case["dr"]).cpu().numpy())
    state = {"case": case, "grid": g, "names": [n for n in case.get("obs", "").split(",") if n]}
    if case["kind"] == "imag":
        state["psi"] = [_device_state(p, case["precision"]) for p in d["psi"]]
    else:
        state["psi"] = _device_state(d["psi"], case["precision"])
    for key in ("field", "alpha"):
        if key in d:
            state[key] = d[key]
    if case["kind"] == "adjoint":
        state["weight"] = (_radius2(shape, case["dr"]) > case["radius"] ** 2).to(torch.float64).cpu().numpy()
    torch.cuda.synchronize()  # the grid works on a stream of its own
    return state


def _rows(rows, precision):
    """Observables of a mixed-precision run carry the rounding of its FP32 state: they go back in that
    type."""
    if isinstance(rows, torch.Tensor):
        return rows if precision == "fp64" else rows.to(torch.float32)
    return rows if precision == "fp64" else rows.astype(np.float32)


def run(state):
    case = state["case"]
    kind, precision = case["kind"], case["precision"]
    if kind == "sweep":
        launch(state["runs"])
        return {"psi": [r[1] for r in state["runs"]], "rows": [_rows(r[3], precision) for r in state["runs"]]}
    g, psi = state["grid"], state["psi"]
    if kind == "imag":
        for j in range(len(psi)):
            g.imag_propagate(psi, j, case["steps"])
        return {"psi": psi, "energies": _rows(np.stack([g.energies(p, 2) for p in psi]), precision)}
    if kind == "length":
        rows = g.run_length(psi, state["field"], state["names"])
        return {"psi": psi, "rows": _rows(rows, precision)}
    if kind == "velocity":
        rows = g.run_velocity(psi, state["field"], state["alpha"], state["names"])
        return {"psi": psi, "rows": _rows(rows, precision)}
    if kind == "step":
        g.integration_step_length(psi, state["field"])
        return {"psi": psi}
    if kind == "adjoint":
        E = torch.tensor(state["field"], requires_grad=True)
        J = length_gauge_objective(g, psi, E, state["weight"], case["checkpoint"])
        J.backward()
        return {"J": J.detach(), "grad": E.grad}
    obs = g.observables(psi, state["names"], state["alpha"])
    dim = len(_shape(case))
    ped, counts, pmd = g.final_spectra(psi, (4.0, 8.0), [case["prmax"]] * dim, case["de"], case["ne"])
    return {"obs": obs, "ped": ped, "counts": counts, "pmd": pmd}


def work(case):
    """The states, potentials, samples and rows in and out once; the transforms a step needs (an FFT of
    N points at 5 N log2 N), its point-wise factors and reductions."""
    if case["kind"] == "sweep":
        parts = [dict(case, kind="length", shape=f"{n}x{n}", integrator="BM4" if k % 2 == 0 else "Verlet")
                 for k, n in enumerate([256] * case["n256"] + [512] * case["n512"] + [1024] * case["n1024"])]
        ws = [work(p) for p in parts]
        return {"bytes": sum(w["bytes"] for w in ws), "flops": sum(w["flops"] for w in ws)}
    shape = _shape(case)
    n = math.prod(shape)
    b = 16 if case["precision"] == "fp64" else 8
    s, steps, kind = len(COEFFICIENTS[case["integrator"]]), case["steps"], case["kind"]
    fft = 5.0 * n * math.log2(n)
    point = 6.0 * n  # one complex factor per point
    substeps = steps * s
    if kind == "imag":
        k = case["states"]
        return {"bytes": 2 * n * b * k + 8 * n, "flops": k * substeps * (2 * fft + 2 * 2 * n) + steps * 16.0 * n * k * (k + 1) / 2}
    if kind in ("length", "velocity"):
        nobs = len(case["obs"].split(",")) * 3.0
        return {"bytes": 2 * n * b + 16 * n, "flops": substeps * (2 * fft + 2 * point) + steps * n * (3 + 2 * nobs)}
    if kind == "step":
        return {"bytes": 2 * n * b + 16 * n, "flops": substeps * (2 * fft + 3 * point)}
    if kind == "adjoint":
        return {"bytes": 2 * n * b + 24 * n, "flops": 3 * substeps * (2 * fft + 2 * point) + substeps * 8.0 * n}
    return {"bytes": n * b + 8 * n + 16.0 * n, "flops": 6 * fft + 20.0 * n * 20}


# ---------------------------------------------------------------- the same in 64 bits with plain torch


class _Plain:
    """The split-operator formulas on complex128 tensors with torch.fft."""

    def __init__(self, case, shape, cap):
        self.shape, self.dr, self.dim = shape, case["dr"], len(shape)
        self.dNr = case["dr"] ** self.dim
        self.as_ = _as(case["integrator"])
        self.s = len(self.as_) // 2
        self.V = _potential(case, shape)
        self.cap = cap
        self.x = [_spread(a, j, self.dim) for j, a in enumerate(_axes(shape, case["dr"]))]
        self.p = [_spread(2 * math.pi * torch.fft.fftfreq(n, case["dr"], dtype=torch.float64, device="cuda"), j, self.dim)
                  for j, n in enumerate(shape)]
        self.kin = 0.5 * sum(p * p for p in self.p)

    def kinetic(self, psi, factor):
        return torch.fft.ifftn(factor * torch.fft.fftn(psi))

    def potential(self, h, E=None):
        v = self.V if E is None else self.V + sum(x * E[j] for j, x in enumerate(self.x))
        f = torch.exp(-1j * h * v)
        return f if self.cap is None else f * torch.exp(-h * self.cap)

    def length_step(self, psi, E):
        a, s = self.as_, self.s
        for i in range(s):
            psi = self.kinetic(psi, torch.exp(-1j * (a[0] if i == 0 else a[2 * i - 1] + a[2 * i]) * self.kin))
            psi = self.potential(a[2 * i] + a[2 * i + 1], E[i]) * psi
        return self.kinetic(psi, torch.exp(-1j * a[2 * s - 1] * self.kin))

    def velocity_step(self, psi, A):
        a = self.as_
        for i in range(self.s):
            psi = self.potential(a[2 * i]) * psi
            h = a[2 * i] + a[2 * i + 1]
            kin = sum(0.5 * p * p + (p + 0.5 * float(A[i][j])) * float(A[i][j]) for j, p in enumerate(self.p))
            psi = self.potential(a[2 * i + 1]) * self.kinetic(psi, torch.exp(-1j * h * kin))
        return psi

    def imag_step(self, psi):
        a = self.as_
        for i in range(self.s):
            psi = torch.exp(-a[2 * i] * self.V) * psi
            psi = torch.exp(-a[2 * i + 1] * self.V) * self.kinetic(psi, torch.exp(-(a[2 * i] + a[2 * i + 1]) * self.kin))
        return psi

    def energy_moment(self, psi):
        return self.kinetic(psi, self.kin) + self.V * psi

    def observables(self, psi, names, alpha=None):
        rho = psi.abs() ** 2
        out = []
        for name in names:
            if name == "norm":
                out.append(rho.sum() * self.dNr)
            elif name == "dipole_r":
                out += [(x * rho).sum() * self.dNr for x in self.x]
            elif name == "accel":
                r2 = _radius2(self.shape, self.dr)
                out += [-(x / (r2 + 0.64) ** 1.5 * rho).sum() * self.dNr for x in self.x]
            elif name == "dipole_v":
                # the unitary momentum density summed with the momentum cell, as the parameter files' runs do
                dNp = math.prod(2 * math.pi / (n * self.dr) for n in self.shape)
                k2 = torch.fft.fftn(psi).abs() ** 2 * (dNp / psi.numel())
                out += [((p + float(alpha[j])) * k2).sum() for j, p in enumerate(self.p)]
            elif name == "energy":
                out.append((psi.conj() * self.energy_moment(psi)).sum().real * self.dNr)
            elif name == "Lz":
                if self.dim == 1:
                    out.append(torch.zeros((), dtype=torch.float64, device="cuda"))
                else:
                    py = self.kinetic(psi, self.p[1] + float(alpha[1]))
                    px = self.kinetic(psi, self.p[0] + float(alpha[0]))
                    out.append((psi.conj() * (self.x[0] * py - self.x[1] * px)).sum().real * self.dNr)
        return torch.stack(out)


def exact(case, seed):
    if case["kind"] == "sweep":
        psis, rows = [], []
        for m, psi, E in _members(case, seed):
            shape = _shape(m)
            L = [0.5 * n * m["dr"] - 5.0 for n in shape]
            cap = sum(0.05 * torch.clamp(_spread(a, j, 2).abs() - L[j], min=0.0) ** 2
                      for j, a in enumerate(_axes(shape, m["dr"])))
            q, r = _Plain(m, shape, cap), []
            for k in range(m["steps"]):
                psi = q.length_step(psi, E[k])
                r.append(q.observables(psi, m["obs"].split(",")))
            psis.append(psi)
            rows.append(torch.stack(r))
        return {"psi": psis, "rows": rows}
    d = _inputs(case, seed)
    kind, names = case["kind"], [n for n in case.get("obs", "").split(",") if n]
    q = _Plain(case, d["shape"], None if kind in ("imag", "spectra") else _vcap(d["shape"], case["dr"]))
    psi = d["psi"]
    if kind == "imag":
        done, energies = [], []
        for p in psi:
            for _ in range(case["steps"]):
                p = q.imag_step(p)
                for o in done:
                    p = p - (o.conj() * p).sum() * q.dNr * o
                p = p / torch.sqrt((p.abs() ** 2).sum() * q.dNr)
            done.append(p)
        for p in done:
            h1 = q.energy_moment(p)
            h2 = q.energy_moment(h1)
            energies.append(torch.stack([(p.conj() * h).sum().real * q.dNr for h in (h1, h2)]))
        return {"psi": done, "energies": torch.stack(energies)}
    if kind in ("length", "velocity"):
        rows = []
        for k in range(case["steps"]):
            rows.append(q.observables(psi, names))
            psi = (q.length_step if kind == "length" else q.velocity_step)(psi, d["field"][k])
        return {"psi": psi, "rows": torch.stack(rows)}
    if kind == "step":
        root = math.sqrt(psi.numel())
        return {"psi": torch.fft.fftn(q.length_step(torch.fft.ifftn(psi) * root, d["field"][0])) / root}
    if kind == "adjoint":
        E = torch.tensor(d["field"], device="cuda", requires_grad=True)
        for k in range(case["steps"]):
            psi = q.length_step(psi, E[k])
        J = (psi.abs() ** 2)[(_radius2(d["shape"], case["dr"]) > case["radius"] ** 2).expand(d["shape"])].sum() * q.dNr
        J.backward()
        return {"J": J.detach(), "grad": E.grad}
    obs = q.observables(psi, names, d["alpha"])
    r = torch.sqrt(_radius2(d["shape"], case["dr"]))
    ramp = torch.sin(0.5 * math.pi * (r - 4.0) / 4.0) ** 2
    f = torch.where(r > 8.0, 1.0, torch.where(r >= 4.0, ramp, 0.0))
    k = torch.fft.fftn(f * psi) / math.sqrt(psi.numel())
    keep = torch.ones(d["shape"], dtype=torch.bool, device="cuda")
    for p in q.p:
        keep = keep & (p.abs() <= case["prmax"])
    counts = [int((p.abs() <= case["prmax"]).sum()) for p in q.p]
    kk, kin = k[keep], q.kin.expand(d["shape"])[keep]
    de, w = case["de"], kk.abs() ** 2
    ped = torch.stack([(w * torch.exp(-0.5 * ((kin - j * de) / de) ** 2)).sum() for j in range(case["ne"])])
    ped = ped / (2 * math.pi * de * de) ** (0.5 * q.dim)
    return {"obs": obs, "ped": ped, "counts": counts, "pmd": torch.stack([w, torch.angle(kk)], dim=1)}
