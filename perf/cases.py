"""The work whose speed this framework is judged by: reacting-flow steps,
their parts and their derivatives, through the public entry points, over the
sizes, boundary sets, flux options and precisions that its examples, tests
and benchmark use.

``listed()`` names twelve cases, ``draw(rng)`` makes more of the same ranges,
``prepare`` builds the state a program holds before the call, ``run`` is one
pass, ``exact`` restates the pass in plain float64 torch (the gas tables are
input data, as a mechanism file is), and ``work`` counts what a pass cannot
do without.
"""
import functools
import math

import numpy as np
import torch

from janc_b200 import mechanism as _mech
from janc_b200.adjoint import Trajectory, probe_trajectory
from janc_b200.ensemble import Ensemble
from janc_b200.solver import Solver

ATM = 101325.0
DX_TUBE = 5e-5           # 1D tubes
DX_CHANNEL = 0.2 / 1024  # 2D channel
RDC_SCALES = {"P0": 10 * ATM, "T0": 300, "R0": 369, "x0": 0.08}
TRANSPORT = {"viscosity_model": "Sutherland", "thermal_conductivity_model": "Prandtl number", "Pr": 0.72,
             "species_diffusivity_model": "Lewis number", "Le": 1.0}
SIDES = ("left_boundary", "right_boundary", "bottom_boundary", "top_boundary")
BOUNDARIES = {
    "tube": ("slip_wall", "zero_gradient", "slip_wall", "slip_wall"),
    "walls": ("slip_wall", "slip_wall", "slip_wall", "slip_wall"),
    "outlet": ("slip_wall", "pressure_outlet", "slip_wall", "slip_wall"),
    "noslip": ("no_slip_wall", "zero_gradient", "no_slip_wall", "no_slip_wall"),
    "periodic": ("slip_wall", "zero_gradient", "periodic", "periodic"),
    "rdc": ("periodic", "periodic", "rdc_injector", "pressure_outlet"),
}


@functools.lru_cache(maxsize=None)
def _mechanism(scaled=False):
    return _mech.load(_mech.DEFAULT_MECHANISM, RDC_SCALES if scaled else None)


def listed():
    return [
        # the smallest runs: a short 1D tube stepped a few steps a call, where
        # launches and latency are what a user waits for
        _step("tube_small_fp64", 1, 500, 1, "fp64", "tube", 4),
        # the longest 1D tubes of the ensemble's range, with an outlet
        _step("tube_long_mixed", 1, 12000, 1, "mixed", "outlet", 4),
        # the benchmark channel, in the fast variant and in float64
        _step("channel_mixed", 2, 1024, 256, "mixed", "walls", 2),
        _step("channel_fp64", 2, 1024, 256, "fp64", "walls", 2),
        # the largest: the rotating-detonation annulus (injector, outlet, ring)
        _step("annulus_mixed", 2, 1600, 1000, "mixed", "rdc", 1),
        # the Godunov path on an odd-sized grid
        _step("hllc_fp64_odd", 2, 517, 251, "fp64", "periodic", 1, flux="HLLC"),
        # Navier-Stokes step with walls that hold the gas
        _step("viscous_mixed", 2, 512, 256, "mixed", "noslip", 1, viscous=True),
        # right-hand side alone, for a program with its own time stepping
        {"name": "rhs_fp64_odd", "op": "rhs", "dim": 2, "nx": 1001, "ny": 333, "precision": "fp64",
         "boundary": "outlet", "flux": "LF", "recon": "WENO5_JS", "viscous": False},
        # chemistry and temperature alone, for a program with its own splitting
        {"name": "chemistry_fp64", "op": "chemistry", "dim": 2, "nx": 700, "ny": 301, "precision": "fp64"},
        # the batched parameter study: many tubes in one launch
        {"name": "ensemble_mixed", "op": "ensemble", "tubes": 64, "lo": 1000, "hi": 16000, "precision": "mixed",
         "steps": 4},
        # gradients of a probe pressure: forward with checkpoints and backward
        {"name": "adjoint_fp64", "op": "adjoint", "nx": 200, "ny": 96, "steps": 6, "checkpoint": 3},
        # one level of a block-structured grid
        {"name": "blocks_fp64", "op": "blocks", "nb": 300, "bx": 20, "by": 20, "recon": "WENO5_JS"},
    ]


def _step(name, dim, nx, ny, precision, boundary, steps, flux="LF", recon="WENO5_JS", viscous=False):
    c = {"op": "step", "dim": dim, "nx": nx, "ny": ny, "precision": precision, "boundary": boundary, "steps": steps,
         "flux": flux, "recon": recon, "viscous": viscous}
    if name:
        c["name"] = name
    return c


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["tube", "tube", "channel", "channel", "channel", "annulus", "godunov", "options", "viscous", "rhs",
                     "chemistry", "ensemble", "adjoint", "blocks"])
    precision = rng.choice(["mixed", "fp64"])
    if op == "tube":
        return _step(None, 1, _log_int(rng, 200, 16000), 1, precision, rng.choice(["tube", "outlet", "noslip"]),
                     rng.randint(1, 6))
    if op == "ensemble":
        lo = _log_int(rng, 300, 2000)
        return {"op": "ensemble", "tubes": rng.randint(4, 64), "lo": lo, "hi": lo * rng.randint(2, 8),
                "precision": precision, "steps": rng.randint(1, 4)}
    if op == "blocks":
        return {"op": "blocks", "nb": _log_int(rng, 16, 500), "bx": rng.randint(8, 24), "by": rng.randint(8, 24),
                "recon": rng.choice(["WENO5_JS", "WENO5_JS", "MUSCL"])}
    if op == "adjoint":
        return {"op": "adjoint", "nx": _log_int(rng, 24, 256), "ny": _log_int(rng, 16, 96), "steps": rng.randint(2, 6),
                "checkpoint": rng.randint(2, 4)}
    cells = _log_int(rng, 3000, 1500000 if op in ("channel", "annulus", "chemistry") else 400000)
    ny = max(8, int(round(math.sqrt(cells * rng.uniform(0.15, 1.2)))))
    nx = max(8, cells // ny)
    walls = rng.choice(["walls", "tube", "outlet", "noslip", "periodic"])
    if op == "annulus":
        return _step(None, 2, nx, ny, precision, "rdc", 1)
    if op == "channel":
        return _step(None, 2, nx, ny, precision, walls, 1 if cells > 200000 else rng.randint(1, 3))
    if op == "godunov":
        return _step(None, 2, nx, ny, precision, walls, 1, flux=rng.choice(["HLLC", "HLLC", "AUSMPW_plus"]))
    if op == "options":
        flux, recon = rng.choice([("LF", "MUSCL"), ("SW", "WENO5_JS"), ("HLLC", "MUSCL")])
        return _step(None, 2, nx, ny, precision, walls, 1, flux=flux, recon=recon)
    if op == "viscous":
        return _step(None, 2, nx, ny, precision, walls, 1, viscous=True)
    if op == "rhs":
        return {"op": "rhs", "dim": 2, "nx": nx, "ny": ny, "precision": precision, "boundary": walls, "flux": "LF",
                "recon": "WENO5_JS", "viscous": False}
    return {"op": "chemistry", "dim": 2, "nx": nx, "ny": ny, "precision": "fp64"}


# ------------------------------------------------------------- initial fields
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _rand(gen, *shape):
    return torch.rand(shape, generator=gen, dtype=torch.float64, device="cuda")


def _burnt():
    """Hot products with their radicals (H2, O2, O, H, OH, HO2, H2O2, H2O by
    the mechanism's names), the rest nitrogen."""
    y = {"H2": 0.0035, "O2": 0.012, "O": 0.0022, "H": 0.0004, "OH": 0.016, "HO2": 6e-6, "H2O2": 8e-7, "H2O": 0.215}
    return torch.tensor([y[s] for s in _mechanism().species[:8]], dtype=torch.float64, device="cuda")


def _wave_fields(gen, shape, mech, floor=0.0, phi=1.0):
    """A detonation on its way through the domain: burnt gas at the left, a
    shocked induction zone, and fresh gas at rest with 1 % of noise; the front
    lies at a seeded place and is wrinkled in 2D.  (P, T, Y, velocities)."""
    nx = shape[0]
    ny = shape[1] if len(shape) == 2 else 1
    x = torch.arange(nx, dtype=torch.float64, device="cuda")[:, None] / nx
    y = torch.arange(ny, dtype=torch.float64, device="cuda")[None, :] / ny
    place = 0.25 + 0.3 * _rand(gen, 1)
    front = place + torch.zeros_like(y)
    for k in range(1, 5):
        r = _rand(gen, 2)
        front = front + 0.03 * (r[0] - 0.5) * torch.cos(2 * math.pi * (k * y + r[1])) * (ny > 1)
    shock = torch.sigmoid((front + 0.06 - x) * nx / 1.2)   # 1 behind the shock
    flame = torch.sigmoid((front - x) * nx / 2.5)          # 1 in the burnt gas
    wave = 0.02 * torch.sin(9 * math.pi * x + 6 * _rand(gen, 1)) * torch.cos(2 * math.pi * y)
    noise = 0.01 * (2 * _rand(gen, 2, nx, ny) - 1)
    P = ATM * (1 + 21 * shock - 6 * flame) * (1 + noise[0] + shock * wave)
    T = (300 + 1150 * shock + 1500 * flame) * (1 + noise[1] + flame * wave)
    fresh = torch.as_tensor(_mech.stoichiometric_Y(mech, phi), device="cuda")
    burnt = _burnt()
    tail = flame[None] * (1 + 0.05 * (2 * _rand(gen, 8, 1, 1) - 1))
    Y = fresh[:, None, None] * (1 - flame[None]) + burnt[:, None, None] * tail
    if floor:
        Y = Y + floor * (1 + _rand(gen, 8, nx, ny))
    u = (900 * shock - 300 * flame) * (1 + noise[1]) + 4 * noise[0]
    v = 60 * shock * torch.sin(2 * math.pi * (2 * y + _rand(gen, 1))) * (ny > 1) + 4 * noise[1]
    out = [P[None], T[None], Y, u[None], v[None]]
    if len(shape) == 1:
        out = [f[..., 0].contiguous() for f in out[:4]]
        return out[0], out[1], out[2], [out[3]]
    return out[0], out[1], out[2].contiguous(), [out[3], out[4]]


def _annulus_fields(gen, nx, ny):
    """The unrolled annulus of the rotating-detonation example, in its own
    scales: a fresh layer over the injector plane, a hot kernel in it, air
    above, all with 1 % of noise.  (P, T, Y, velocities, Yinj)."""
    s = RDC_SCALES
    a = 1.0 / 8 * 0.232
    y_h2, y_o2 = a / (1 + a), 0.232 / (1 + a)
    env = torch.tensor([0, 0.232, 0, 0, 0, 0, 0, 0.0], dtype=torch.float64, device="cuda")
    fill = torch.tensor([y_h2, y_o2, 0, 0, 0, 0, 0, 0.0], dtype=torch.float64, device="cuda")
    x = torch.arange(nx, dtype=torch.float64, device="cuda")[:, None] / nx
    y = torch.arange(ny, dtype=torch.float64, device="cuda")[None, :] / ny
    layer = torch.sigmoid((0.36 * (1 - 2 * x) - y) * ny / 2.0)
    hot = torch.sigmoid((0.03 - x) * nx / 2.0) * torch.sigmoid((0.1 - y) * ny / 2.0)
    noise = 0.01 * (2 * _rand(gen, 4, nx, ny) - 1)
    Y = env[:, None, None] * (1 - layer[None]) + fill[:, None, None] * layer[None]
    Y = Y * (1 - 0.6 * hot[None]) + 0.6 * hot[None] * _burnt()[:, None, None]
    P = (0.1 + (3.0 + 2 * _rand(gen, 1)) * hot) * (1 + noise[0])
    T = (1.0 + 8.5 * hot) * (1 + noise[1])
    u0 = math.sqrt(s["R0"] * s["T0"])
    vel = [((60 * layer + 300 * hot) / u0 * (1 + noise[2]))[None], ((120 * layer) / u0 * (1 + noise[3]))[None]]
    yinj = np.concatenate([[y_h2, y_o2], 1e-20 * np.ones(6)])
    return P[None], T[None], Y.contiguous(), vel, yinj


def _fields(case, seed):
    """(mechanism, nondim config, P, T, Y, velocities, theta) of a case."""
    gen = _generator(seed)
    shape = (case["nx"],) if case.get("dim", 2) == 1 else (case["nx"], case["ny"])
    if case.get("boundary") == "rdc":
        mech = _mechanism(True)
        P, T, Y, vel, yinj = _annulus_fields(gen, *shape)
        return mech, P, T, Y, vel, {"Pb": 0.1, "Yinj": yinj}
    mech = _mechanism()
    P, T, Y, vel = _wave_fields(gen, shape, mech, floor=2e-6 if case["op"] == "adjoint" else 0.0)
    return mech, P, T, Y, vel, {"Pb": ATM} if case.get("boundary") == "outlet" else None


def _spacing(case):
    if case.get("boundary") == "rdc":
        return 1.0 / 400
    return DX_TUBE if case.get("dim", 2) == 1 else DX_CHANNEL


def _cfl(case):
    return 0.05 if case.get("dim", 2) == 2 and case.get("boundary") != "rdc" else 0.1


def _boundaries(case):
    return dict(zip(SIDES[: 2 * case.get("dim", 2)], BOUNDARIES[case.get("boundary", "walls")]))


def _flux_config(case):
    c = {"interface_reconstruction": case["recon"], "viscosity": "on" if case["viscous"] else "off"}
    if case["flux"] in ("LF", "SW"):
        return dict(c, solver_type="flux_splitting", split_method=case["flux"])
    return dict(c, solver_type="godunov", riemann_solver=case["flux"])


def _tubes(case, seed):
    """(nx list, [(U, aux)]) of an ensemble: lengths over the range, an
    equivalence ratio and a front for each."""
    rng = np.random.default_rng(seed)
    mech = _mechanism()
    gas = Gas(mech)
    n = case["tubes"]
    # the lengths are the case's, not the seed's: the same study on new states
    grid = (np.arange(n) + 0.5) / n
    nxs = [int(v) for v in np.round(case["lo"] * (case["hi"] / case["lo"]) ** grid)]
    states = []
    for nx, phi in zip(nxs, rng.uniform(0.6, 1.4, n)):
        P, T, Y, vel = _wave_fields(_generator(rng.integers(1 << 30)), (nx,), mech, phi=float(phi))
        states.append(gas.state(P, T, Y, vel))
    return mech, nxs, states


def _block_data(case, seed):
    """Ghost-padded blocks (nb, 14, bx + 6, by + 6): windows of one field."""
    nb, X, Y_ = case["nb"], case["bx"] + 6, case["by"] + 6
    mech = _mechanism()
    gas = Gas(mech)
    side = int(math.ceil(math.sqrt(nb)))
    P, T, Y, vel = _wave_fields(_generator(seed), (side * case["bx"] + 6, side * case["by"] + 6), mech)
    U, aux = gas.state(P, T, Y, vel)
    g = torch.cat([U, aux], 0).unfold(1, X, case["bx"]).unfold(2, Y_, case["by"])  # (14, side, side, X, Y)
    return mech, g.permute(1, 2, 0, 3, 4).reshape(side * side, 14, X, Y_)[:nb].contiguous()


BLOCK_DT = 2e-9


def prepare(case, seed):
    op = case["op"]
    if op == "ensemble":
        mech, nxs, states = _tubes(case, seed)
        ens = Ensemble(nxs, DX_TUBE, cfl=0.1, precision=case["precision"])
        live = [t for i in range(len(nxs)) for t in ens.state(i)]
        return {"case": case, "ens": ens, "live": live, "start": [t for s in states for t in s]}
    if op == "blocks":
        mech, G = _block_data(case, seed)
        s = Solver(2, 32, 32, DX_CHANNEL, DX_CHANNEL, _boundaries(case), mech, precision="fp64",
                   flux_config={"solver_type": "flux_splitting", "split_method": "LF",
                                "interface_reconstruction": case["recon"], "viscosity": "off"})
        return {"case": case, "solver": s, "G": G}
    mech, P, T, Y, vel, theta = _fields(case, seed)
    d = _spacing(case)
    if op == "adjoint":
        s = Solver(2, case["nx"], case["ny"], d, d, _boundaries(case), mech, precision="fp64")
        traj = Trajectory(s, cfl=0.05, probe=_probe(case), checkpoint=case["checkpoint"])
        return {"case": case, "solver": s, "traj": traj, "P": P.contiguous(), "T": T.contiguous(), "Y": Y}
    U, aux = Gas(mech).state(P, T, Y, vel)
    if op == "chemistry":
        s = Solver(2, case["nx"], case["ny"], d, d, _boundaries(case), mech, precision=case["precision"])
        return {"case": case, "solver": s, "U": U, "aux": aux}
    dim = case["dim"]
    s = Solver(dim, case["nx"], case["ny"] if dim == 2 else None, d, d if dim == 2 else None, _boundaries(case), mech,
               precision=case["precision"], flux_config=_flux_config(case),
               transport_config=TRANSPORT if case["viscous"] else None)
    return {"case": case, "solver": s, "U": U, "aux": aux, "theta": theta}


def _probe(case):
    return (int(0.5 * case["nx"]), case["ny"] // 2, 4, 4)


CHEM_DT = 4e-9
RHS_DT = 4e-9


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "step":
        U, aux, dts = state["solver"].advance(state["U"], state["aux"], case["steps"], cfl=_cfl(case),
                                              theta=state["theta"])
        return {"U": U, "aux": aux, "dt": dts}
    if op == "rhs":
        return state["solver"].flux_func(state["U"], state["aux"], dt=RHS_DT, theta=state["theta"])
    if op == "chemistry":
        s = state["solver"]
        S = s.reaction_source_terms(state["U"], state["aux"], CHEM_DT)
        return {"S": S, "aux": s.update_aux(state["U"] + S, state["aux"])}
    if op == "ensemble":
        ens = state["ens"]
        torch._foreach_copy_(state["live"], state["start"])
        dts = ens.advance(case["steps"], record_dt=True)
        return {"U": torch.cat(state["live"][0::2], 1), "aux": torch.cat(state["live"][1::2], 1), "dt": dts}
    if op == "adjoint":
        T = state["T"].detach().clone().requires_grad_()
        ln_a = torch.zeros(19, dtype=torch.float64, device=T.device, requires_grad=True)
        dts, pps = probe_trajectory(state["traj"], state["P"], T, state["Y"], ln_a, case["steps"])
        (dts * pps).sum().backward()
        return {"dt": dts.detach(), "p": pps.detach(), "T_grad": T.grad, "lnA_grad": ln_a.grad}
    s, G = state["solver"], state["G"]
    B1 = s.amr_stage(G, None, 1, DX_CHANNEL, DX_CHANNEL, BLOCK_DT)
    B2 = s.amr_stage(B1, G, 2, DX_CHANNEL, DX_CHANNEL, BLOCK_DT)
    B3 = s.amr_stage(B2, G, 3, DX_CHANNEL, DX_CHANNEL, BLOCK_DT)
    return s.amr_chem(B3[..., 3:-3, 3:-3].contiguous(), BLOCK_DT)


# Operations of one cell: WENO5 of one field at one face from both sides with
# its splitting (about 150), the state's combination and temperature (350),
# face thermodynamics and solver of a Godunov face (600), node derivatives and
# transport of the viscous part (700), the chemistry of one cell (6800).
def work(case):
    op = case["op"]
    if op == "ensemble":
        n = case["tubes"]
        cells = sum(round(case["lo"] * (case["hi"] / case["lo"]) ** ((i + 0.5) / n)) for i in range(n))
        return {"bytes": 2 * 13 * 8 * cells, "flops": cells * case["steps"] * (3 * (11 * 150 + 350) + 6800)}
    if op == "blocks":
        cells = case["nb"] * case["bx"] * case["by"]
        padded = case["nb"] * (case["bx"] + 6) * (case["by"] + 6)
        return {"bytes": 14 * 8 * (padded + cells), "flops": cells * (3 * (24 * 150 + 350) + 6800)}
    cells = case["nx"] * case.get("ny", 1)
    if op == "adjoint":
        # forward, its recomputation, and a reverse sweep of about twice a step
        return {"bytes": 8 * 11 * cells, "flops": 4 * cells * case["steps"] * (3 * (24 * 150 + 350) + 6800)}
    if op == "chemistry":
        return {"bytes": 8 * cells * (14 + 12 + 2), "flops": cells * 7150}
    dim = case["dim"]
    fields = 10 + dim
    rhs = dim * (fields * 150 + (600 if case["flux"] in ("HLLC", "AUSMPW_plus") else 0)) + (
        700 if case["viscous"] else 0)
    if op == "rhs":
        return {"bytes": 8 * cells * (2 * fields + 2), "flops": cells * rhs}
    return {"bytes": 2 * (fields + 2) * 8 * cells, "flops": cells * case["steps"] * (3 * (rhs + 350) + 6800)}


# ------------------------------------------------ the same in plain float64
def _poly(c, x):
    r = torch.full_like(x, c[0])
    for a in c[1:]:
        r = r * x + a
    return r


class Gas:
    """Ideal-gas mixture of NASA7 species with point-implicit kinetics."""

    def __init__(self, mech):
        t = mech.tables
        self.t = {k: np.asarray(v, dtype=np.float64).tolist() for k, v in t.items()}
        self.M, self.Tc = self.t["species_M"], self.t["Tcr"]
        self.T0, self.P0 = float(mech.scales.T0), float(mech.scales.P0)
        self.lnA = None  # offsets of ln A

    @staticmethod
    def full(Y):
        return torch.cat([Y, 1 - Y.sum(0, keepdim=True)], 0)

    def R(self, Y):
        return sum(y / m for y, m in zip(self.full(Y), self.M))[None]

    def _species(self, name, T, k):
        return torch.where(T < self.Tc[k], _poly(self.t[name % "low"][k], T), _poly(self.t[name % "high"][k], T))

    def thermo(self, T, Y):
        """cp, h, dcp/dT of the mixture; T (1, ...)."""
        F = self.full(Y)
        return [sum(self._species(n, T, k) * F[k] for k in range(9))
                for n in ("cp_cof_%s", "h_cof_%s", "dcp_cof_%s")]

    def state(self, P, T, Y, vel):
        cp, h, _ = self.thermo(T, Y)
        R = self.R(Y)
        rho = P / (R * T)
        E = rho * h - P + 0.5 * rho * sum(v * v for v in vel)
        U = torch.cat([rho] + [rho * v for v in vel] + [E, rho * Y], 0).contiguous()
        return U, torch.cat([cp / (cp - R), T], 0).contiguous()

    def split(self, U):
        """rho, velocities, E / rho, Y"""
        d = U.shape[0] - 10
        rho = U[0:1]
        return rho, [U[1 + i:2 + i] / rho for i in range(d)], U[1 + d:2 + d] / rho, U[2 + d:] / rho

    def temperature(self, U, aux, grad=False):
        rho, vel, E, Y = self.split(U)
        e = E - 0.5 * sum(v * v for v in vel)
        R = self.R(Y)
        T = aux[1:2].detach()
        with torch.no_grad():
            for _ in range(6):
                cp, h, dcp = self.thermo(T, Y)
                res, d1 = h - R * T - e, cp - R
                if not float(res.abs().max()) > 5e-9 or _ == 5:
                    break
                T = T - 2 * res * d1 / (2 * d1 * d1 - res * dcp)
        cp, h, _ = self.thermo(T, Y)
        if grad:  # the implicit derivative of h - R T = e at the solution
            res = h - R * T - e
            T = T - (res - res.detach()) / (cp - R).detach()
            cp = self.thermo(T, Y)[0]
        return torch.cat([cp / (cp - R), T], 0)

    def prims(self, U, aux):
        rho, vel, _, Y = self.split(U)
        p = rho * self.R(Y) * aux[1:2]
        return rho, vel, Y, p, torch.sqrt(aux[0:1] * p / rho)

    def source(self, U, aux, dt):
        t = self.t
        rho, vel, _, Y8 = self.split(U)
        T = aux[1]
        Y = self.full(Y8)
        X = [rho[0] * Y[k] / self.M[k] for k in range(9)]
        Xc = [x.clamp(min=1e-50) for x in X]
        lX, lT = [torch.log(x) for x in Xc[:8]], torch.log(self.T0 * T)
        g = []
        for k in range(8):
            lo = T < self.Tc[k]
            s = torch.where(lo, _poly(t["s_cof_low"][k], T) + t["logcof_low"][k] * lT,
                            _poly(t["s_cof_high"][k], T) + t["logcof_high"][k] * lT)
            h = torch.where(lo, _poly(t["h_cof_low_chem"][k], T), _poly(t["h_cof_high_chem"][k], T))
            g.append(s - h / T)
        w = [torch.zeros_like(T) for _ in range(8)]
        J = [[torch.zeros_like(T) for _ in range(8)] for _ in range(8)]
        for i in range(len(t["A"])):
            vf, vb, tb = t["vf"][i], t["vb"][i], t["third_body"][i]
            k0 = t["A"][i] * T ** t["B"][i] * torch.exp(-t["EaR"][i] / T)
            if self.lnA is not None:
                k0 = k0 * torch.exp(self.lnA[i])
            third = t["is_third_body"][i] > 0
            Mi = sum(a * x for a, x in zip(tb, X) if a) if third else torch.ones_like(T)
            sf = sum(v * l for v, l in zip(vf, lX) if v)
            sb = sum(v * l for v, l in zip(vb, lX) if v)
            sg = sum((b - f) * q for f, b, q in zip(vf, vb, g) if b != f)
            kf = k0 * torch.exp(sf)
            kb = k0 / (torch.exp(sg) * (ATM / self.P0 / T) ** t["vsum"][i]) * torch.exp(sb)
            dq = kf - kb
            for k in range(8):
                dv = vb[k] - vf[k]
                if dv == 0:
                    continue
                w[k] = w[k] + dv * Mi * dq
                for n in range(8):
                    if third and tb[n]:
                        J[k][n] = J[k][n] + dv * dq * (tb[n] / self.M[n])
                    if vf[n] or vb[n]:
                        J[k][n] = J[k][n] + dv * Mi * (vf[n] * kf - vb[n] * kb) / (self.M[n] * Xc[n])
        A = torch.stack([torch.stack([(1.0 / dt if k == n else 0.0) - self.M[k] * J[k][n] for n in range(8)], -1)
                         for k in range(8)], -2)
        b = torch.stack([self.M[k] * w[k] for k in range(8)], -1)
        shape = T.shape
        x = torch.linalg.solve(A.reshape(-1, 8, 8), b.reshape(-1, 8, 1))[..., 0].reshape(*shape, 8)
        dY = torch.movedim(x, -1, 0) / rho
        dY = torch.minimum(torch.maximum(dY, -Y8), 1 - Y8)
        return torch.cat([torch.zeros_like(U[:U.shape[0] - 8]), rho * dY], 0)


def _outlet(gas, U, aux, normal, Pb):
    rho, vel, _, Y = gas.split(U)
    R = gas.R(Y)
    p = rho * R * aux[1:2]
    sub = normal / torch.sqrt(aux[0:1] * p / rho) < 1
    rho_c = torch.where(sub, Pb / (p / rho), rho)
    p_c = torch.where(sub, torch.full_like(p, Pb), p)
    T_c = torch.where(sub, p_c / (rho_c * R), aux[1:2])
    return gas.state(p_c, T_c, Y, vel)


def _injector(gas, U, aux, yinj):
    """A choked injector below the first row (area ratios 1 : 4 : 5, total
    pressure and temperature 1), blocked where the pressure is at least 1."""
    rho, vel, Y, p, _ = gas.prims(U, aux)
    Yi = torch.as_tensor(yinj, dtype=torch.float64, device=U.device).reshape(8, *([1] * (U.ndim - 1)))
    Yi = Yi.expand(8, *U.shape[1:])
    R, k = gas.R(Yi), 1.29
    m1, m2 = torch.zeros_like(p), torch.ones_like(p)
    for _ in range(20):
        M = 0.5 * (m1 + m2)
        b = 1 + (k - 1) / 2 * M * M
        P1, V1 = b ** (-k / (k - 1)), M * b ** -0.5 * torch.sqrt(k * R)
        flow = torch.sqrt(k / R) * M * b ** (-(k + 1) / 2 / (k - 1))
        B = k / (k - 1) * p * 5 / flow
        V3 = -B + torch.sqrt(B * B + 2 * k / (k - 1) * R)
        up = (flow * (V3 - V1) - P1 + 5 * p) / 4 >= P1
        m2, m1 = torch.where(up, M, m2), torch.where(up, m1, M)
    T_i = p / (R * (flow / V3 / 5))
    Ui, ai = gas.state(p, T_i, Yi, [torch.zeros_like(p), V3])
    Ub, ab = gas.state(p, aux[1:2], Y, [vel[0], -vel[1]])
    ab = torch.cat([aux[0:1], ab[1:]], 0)
    blk = p >= 1.0
    return torch.where(blk, Ub, Ui), torch.where(blk, ab, ai)


def _pad(gas, U, aux, kinds, theta):
    """Three ghost layers on each side: node-periodic, then each side's own."""
    nv = U.shape[0]
    f = torch.cat([U, aux], 0)
    for ax in range(1, f.ndim):
        n = f.shape[ax]
        i = torch.tensor([n - 4, n - 3, n - 2, *range(n), 1, 2, 3], device=f.device)
        f = f.index_select(ax, i)
    f = f.clone()
    inner = [slice(3, -3)] * (f.ndim - 1)
    for side, kind in enumerate(kinds):
        if kind == "periodic":
            continue
        ax, lo = side // 2, side % 2 == 0
        n = f.shape[1 + ax] - 6

        def at(j):
            s = list(inner)
            s[ax] = slice(j, j + 1)
            return (slice(None), *s)
        for layer in range(3):
            dst = 2 - layer if lo else n + 3 + layer
            copy = kind in ("zero_gradient", "no_slip_wall")
            b = f[at((3 + layer if copy else 3) if lo else (n + 2 - layer if copy else n + 2))].clone()
            if kind == "slip_wall":
                b[1 + ax] = -b[1 + ax]
            elif kind == "no_slip_wall":
                b[1:f.ndim] = -b[1:f.ndim]
            elif kind == "pressure_outlet":
                un = b[1 + ax:2 + ax] / b[0:1]
                b = torch.cat(_outlet(gas, b[:nv], b[nv:], -un if lo else un, theta["Pb"]), 0)
            elif kind == "rdc_injector":
                b = torch.cat(_injector(gas, b[:nv], b[nv:], theta["Yinj"]), 0)
            f[at(dst)] = b
    return f[:nv], f[nv:]


def _weno(a, b, c, d, e):
    s = [13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2,
         13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2,
         13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2]
    q = [a / 3 - 7 / 6 * b + 11 / 6 * c, -b / 6 + 5 / 6 * c + d / 3, c / 3 + 5 / 6 * d - e / 6]
    w = [g / (1e-6 + t) ** 2 for g, t in zip((0.1, 0.6, 0.3), s)]
    return (w[0] * q[0] + w[1] * q[1] + w[2] * q[2]) / (w[0] + w[1] + w[2])


def _minmod(x, y):
    return torch.sign(x) * torch.clamp(torch.minimum(x * torch.sign(y), y * torch.sign(x)), min=0)


def _faces(f, ax, recon):
    """Left and right values at the inner faces along axis ax of an array
    with three ghost layers (the other axes cut to the interior)."""
    for o in range(1, f.ndim):
        if o != ax:
            f = f.narrow(o, 3, f.shape[o] - 6)
    n = f.shape[ax] - 6
    c = [f.narrow(ax, k, n + 1) for k in range(6)]
    if recon == "MUSCL":
        def slope(k, near):
            m, p = c[k] - c[k - 1], c[k + 1] - c[k]
            fw, bw = _minmod(p, m), _minmod(m, p)
            return 0.25 * (2 / 3 * bw + 4 / 3 * fw) if near else 0.25 * (2 / 3 * fw + 4 / 3 * bw)
        return lambda: c[2] + slope(2, True), lambda: c[3] - slope(3, False)
    return lambda: _weno(*c[:5]), lambda: _weno(*c[:0:-1])


def _phys(U, vel, p, ax):
    """Euler flux along ax."""
    d = len(vel)
    F = [U[i:i + 1] * vel[ax] for i in range(U.shape[0])]
    F[1 + ax] = F[1 + ax] + p
    F[1 + d] = F[1 + d] + p * vel[ax]
    return torch.cat(F, 0)


def _steger(U, vel, p, a, gamma, ax):
    d, rho, th = len(vel), U[0:1], vel[ax]
    E = U[1 + d:2 + d]
    x1 = torch.cat([rho] + [U[1 + i:2 + i] - (rho * a if i == ax else 0) for i in range(d)]
                   + [E + p - rho * a * th, U[2 + d:]], 0)
    x4 = torch.cat([rho] + [U[1 + i:2 + i] + (rho * a if i == ax else 0) for i in range(d)]
                   + [E + p + rho * a * th, U[2 + d:]], 0)
    x2 = torch.cat([U[:1 + d], 0.5 * rho * sum(v * v for v in vel), U[2 + d:]], 0)
    out = []
    for sign in (1, -1):
        lam = [0.5 * (q + sign * torch.sqrt(q * q + 1e-12)) for q in (th - a, th, th + a)]
        out.append(lam[0] * x1 / (2 * gamma) + lam[1] * (gamma - 1) / gamma * x2 + lam[2] * x4 / (2 * gamma))
    return out


def _face_state(gas, q):
    """rho, velocities, p, Y, sound speed, rho e (total) and total enthalpy of
    reconstructed primitives [rho, velocities, p, Y]."""
    d = q.shape[0] - 10
    rho, vel, p, Y = q[0:1], [q[1 + i:2 + i] for i in range(d)], q[1 + d:2 + d], q[2 + d:]
    R = gas.R(Y)
    cp, h, _ = gas.thermo(p / (R * rho), Y)
    kin = 0.5 * rho * sum(v * v for v in vel)
    return rho, vel, p, Y, torch.sqrt(cp / (cp - R) * p / rho), rho * h - p + kin, rho * h + kin


def _hllc(gas, qL, qR, ax):
    L, R = _face_state(gas, qL), _face_state(gas, qR)
    uL, uR = L[1][ax], R[1][ax]
    sL, sR = torch.minimum(uL - L[4], uR - R[4]), torch.maximum(uL + L[4], uR + R[4])
    sM = (R[2] - L[2] + L[0] * uL * (sL - uL) - R[0] * uR * (sR - uR)) / (L[0] * (sL - uL) - R[0] * (sR - uR))

    def side(S, s):
        rho, vel, p, Y, _, E, _ = S
        un = vel[ax]
        U = torch.cat([rho] + [rho * v for v in vel] + [E, rho * Y], 0)
        F = _phys(U, vel, p, ax)
        star = [sM if i == ax else v for i, v in enumerate(vel)]
        UM = rho * (s - un) / (s - sM) * torch.cat(
            [torch.ones_like(sM)] + star + [E / rho + (sM - un) * (sM + p / (rho * (s - un))), Y], 0)
        return F, F + s * (UM - U)
    FL, FLM = side(L, sL)
    FR, FRM = side(R, sR)
    F = torch.where(sL >= 0, FL, FR)
    F = torch.where((sL <= 0) & (sM >= 0), FLM, F)
    return torch.where((sM <= 0) & (sR >= 0), FRM, F)


def _ausmpw(gas, qL, qR, ax):
    L, R = _face_state(gas, qL), _face_state(gas, qR)
    c = 0.5 * (L[4] + R[4])
    mL, mR = L[1][ax] / c, R[1][ax] / c
    iL, iR = mL.abs() <= 1, mR.abs() <= 1
    mp = torch.where(iL, 0.25 * (mL + 1) ** 2, 0.5 * (mL + mL.abs()))
    mm = torch.where(iR, -0.25 * (mR - 1) ** 2, 0.5 * (mR - mR.abs()))
    pp = torch.where(iL, 0.25 * (mL + 1) ** 2 * (2 - mL), 0.5 * (1 + torch.sign(mL)))
    pm = torch.where(iR, 0.25 * (mR - 1) ** 2 * (2 + mR), 0.5 * (1 - torch.sign(mR)))
    ps = pp * L[2] + pm * R[2]
    w = 1 - torch.minimum(L[2] / R[2], R[2] / L[2]) ** 3
    fL = torch.where(mL.abs() < 1, L[2] / ps - 1, torch.zeros_like(ps))
    fR = torch.where(mR.abs() < 1, R[2] / ps - 1, torch.zeros_like(ps))
    ind = mp + mm >= 0
    aL = torch.where(ind, mp + mm * ((1 - w) * (1 + fR) - fL), mp * w * (1 + fL))
    aR = torch.where(ind, mm * w * (1 + fR), mm + mp * ((1 - w) * (1 + fL) - fR))
    phi = [torch.cat([S[0]] + [S[0] * v for v in S[1]] + [S[6], S[0] * S[3]], 0) for S in (L, R)]
    F = aL * c * phi[0] + aR * c * phi[1]
    F[1 + ax] = F[1 + ax] + (pp * L[2] + pm * R[2])[0]
    return F


def _slope(f, d, ax):
    """Sixth-order central differences, lower one-sided orders at the ends."""
    n = f.shape[ax]
    s = lambda k, m=1: f.narrow(ax, k, m)  # noqa: E731
    mid = (s(6, n - 6) - s(0, n - 6) + 9 * (s(1, n - 6) - s(5, n - 6)) + 45 * (s(4, n - 6) - s(2, n - 6))) / (60 * d)
    ends = [(s(1) - s(0)) / d, (s(2) - s(0)) / (2 * d), (s(0) - 8 * s(1) + 8 * s(3) - s(4)) / (12 * d)]
    tail = [(s(n - 5) - 8 * s(n - 4) + 8 * s(n - 2) - s(n - 1)) / (12 * d), (s(n - 1) - s(n - 3)) / (2 * d),
            (s(n - 1) - s(n - 2)) / d]
    return torch.cat(ends + [mid] + tail, ax)


def _viscous(gas, U, aux, h):
    rho, vel, Y, _, _ = gas.prims(U, aux)
    T, d = aux[1:2], len(vel)
    cpk = torch.cat([gas._species("cp_cof_%s", T, k) for k in range(9)], 0)
    hk = torch.cat([gas._species("h_cof_%s", T, k) for k in range(9)], 0)
    Yf = gas.full(Y)
    mu = 1.716e-5 * (T / 273.15) ** 1.5 * (273.15 + 110.4) / (T + 110.4)
    kappa = mu * (cpk * Yf).sum(0, keepdim=True) / TRANSPORT["Pr"]
    rhoD = mu * cpk / TRANSPORT["Pr"] / (TRANSPORT["Le"] * cpk)
    grad = [[_slope(v, h, 1 + a) for a in range(d)] for v in vel]
    div = sum(grad[i][i] for i in range(d))
    out = 0
    for ax in range(d):
        tau = [mu * (grad[ax][i] + grad[i][ax]) - (2 / 3 * mu * div if i == ax else 0) for i in range(d)]
        j = -rhoD * _slope(Yf, h, 1 + ax)
        q = -kappa * _slope(T, h, 1 + ax)
        F = torch.cat([torch.zeros_like(rho)] + tau
                      + [sum(v * t for v, t in zip(vel, tau)) - q - (j * hk).sum(0, keepdim=True), -j[:-1]], 0)
        for o in range(1, F.ndim):
            if o != 1 + ax:
                F = F.narrow(o, 3, F.shape[o] - 6)
        n = F.shape[1 + ax] - 6
        c = [F.narrow(1 + ax, k, n + 1) for k in range(6)]
        Fi = (3 * (c[0] + c[5]) - 25 * (c[1] + c[4]) + 150 * (c[2] + c[3])) / 256
        out = out + torch.diff(Fi, dim=1 + ax) / h
    return out


def _rhs(gas, U, aux, h, flux="LF", recon="WENO5_JS", viscous=False):
    """-dF/dx (- dG/dy) of a ghost-padded state."""
    rho, vel, Y, p, a = gas.prims(U, aux)
    out = 0
    for ax in range(len(vel)):
        if flux in ("LF", "SW"):
            F = _phys(U, vel, p, ax)
            if flux == "LF":
                al = (vel[ax].abs() + a).amax()
                hp, hm = 0.5 * (F + al * U), 0.5 * (F - al * U)
            else:
                hp, hm = _steger(U, vel, p, a, aux[0:1], ax)
            F = _faces(hp, 1 + ax, recon)[0]() + _faces(hm, 1 + ax, recon)[1]()
        else:
            left, right = _faces(torch.cat([rho] + vel + [p, Y], 0), 1 + ax, recon)
            F = (_hllc if flux == "HLLC" else _ausmpw)(gas, left(), right(), ax)
        out = out - torch.diff(F, dim=1 + ax) / h
    return out + _viscous(gas, U, aux, h) if viscous else out


def _dt(gas, U, aux, h, cfl):
    _, vel, _, _, a = gas.prims(U, aux)
    return cfl / (sum((v.abs() + a) / h for v in vel)).amax()


def _one_step(gas, U, aux, h, dt, rhs, grad=False):
    """SSP-RK3 of the flux, then the chemistry."""
    U1 = U + dt * rhs(U, aux)
    a1 = gas.temperature(U1, aux, grad)
    U2 = 0.75 * U + 0.25 * (U1 + dt * rhs(U1, a1))
    a2 = gas.temperature(U2, a1, grad)
    U3 = U / 3 + 2 / 3 * (U2 + dt * rhs(U2, a2))
    a3 = gas.temperature(U3, a2, grad)
    U4 = U3 + gas.source(U3, a3, dt)
    return U4, gas.temperature(U4, a3, grad)


def _march(gas, U, aux, h, cfl, steps, kinds, theta, **how):
    dts = []
    for _ in range(steps):
        dt = _dt(gas, U, aux, h, cfl)
        U, aux = _one_step(gas, U, aux, h, dt, lambda q, b: _rhs(gas, *_pad(gas, q, b, kinds, theta), h, **how))
        dts.append(dt)
    return U, aux, torch.stack(dts)


def _exact_gradient(case, seed):
    from torch.utils.checkpoint import checkpoint
    mech, P, T, Y, _, _ = _fields(case, seed)
    h, kinds = _spacing(case), list(_boundaries(case).values())
    x0, y0, wx, wy = _probe(case)
    T = T.clone().requires_grad_()
    ln_a = torch.zeros(19, dtype=torch.float64, device="cuda", requires_grad=True)

    def one(U, aux, lnA):
        gas = Gas(mech)
        gas.lnA = lnA
        dt = _dt(gas, U, aux, h, 0.05)
        U, aux = _one_step(gas, U, aux, h, dt, lambda q, b: _rhs(gas, *_pad(gas, q, b, kinds, None), h), grad=True)
        p = gas.prims(U, aux)[3]
        return U, aux, dt, p[0, x0:x0 + wx, y0:y0 + wy].mean()
    U, aux = Gas(mech).state(P, T, Y, [torch.zeros_like(T)] * 2)
    dts, pps = [], []
    for _ in range(case["steps"]):
        U, aux, dt, p = checkpoint(one, U, aux, ln_a, use_reentrant=False)
        dts.append(dt)
        pps.append(p)
    dts, pps = torch.stack(dts), torch.stack(pps)
    (dts * pps).sum().backward()
    return {"dt": dts.detach(), "p": pps.detach(), "T_grad": T.grad, "lnA_grad": ln_a.grad}


def exact(case, seed):
    op = case["op"]
    if op == "adjoint":
        return _exact_gradient(case, seed)
    with torch.no_grad():
        if op == "ensemble":
            mech, nxs, states = _tubes(case, seed)
            gas = Gas(mech)
            got = [_march(gas, U, aux, DX_TUBE, 0.1, case["steps"], ["slip_wall", "zero_gradient"], None)
                   for U, aux in states]
            return {"U": torch.cat([g[0] for g in got], 1), "aux": torch.cat([g[1] for g in got], 1),
                    "dt": torch.stack([g[2] for g in got])}
        if op == "blocks":
            mech, G = _block_data(case, seed)
            gas = Gas(mech)
            out = []
            for g in G:
                U, aux = g[:12], g[12:]

                def rhs(q, b):
                    r = torch.zeros_like(q)
                    r[:, 3:-3, 3:-3] = _rhs(gas, q, b, DX_CHANNEL, recon=case["recon"])
                    return r
                U1 = U + BLOCK_DT * rhs(U, aux)
                a1 = gas.temperature(U1, aux)
                U2 = 0.75 * U + 0.25 * (U1 + BLOCK_DT * rhs(U1, a1))
                a2 = gas.temperature(U2, a1)
                U3 = U / 3 + 2 / 3 * (U2 + BLOCK_DT * rhs(U2, a2))
                out.append(torch.cat([U3, gas.temperature(U3, a2)], 0)[:, 3:-3, 3:-3])
            B = torch.stack(out, 1)  # (14, nb, bx, by)
            U = B[:12] + gas.source(B[:12].reshape(12, -1, case["by"]), B[12:].reshape(2, -1, case["by"]),
                                    BLOCK_DT).reshape(B[:12].shape)
            flat = U.reshape(12, -1, case["by"])
            aux = gas.temperature(flat, B[12:].reshape(2, -1, case["by"])).reshape(B[12:].shape)
            return torch.cat([U, aux], 0).transpose(0, 1).contiguous()
        mech, P, T, Y, vel, theta = _fields(case, seed)
        gas = Gas(mech)
        U, aux = gas.state(P, T, Y, vel)
        if op == "chemistry":
            S = gas.source(U, aux, CHEM_DT)
            return {"S": S, "aux": gas.temperature(U + S, aux)}
        kinds = list(_boundaries(case).values())
        how = {"flux": case["flux"], "recon": case["recon"], "viscous": case["viscous"]}
        if op == "rhs":
            return RHS_DT * _rhs(gas, *_pad(gas, U, aux, kinds, theta), _spacing(case), **how)
        U, aux, dts = _march(gas, U, aux, _spacing(case), _cfl(case), case["steps"], kinds, theta, **how)
        return {"U": U, "aux": aux, "dt": dts}
