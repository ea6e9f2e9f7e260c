"""Timed workloads of the SLIC solver, each through the package's public entry points.

A case names a model, a grid, the kernel form and the run's options; one pass takes a state that the caller holds
through the whole call (upload, the device time loop, download) and returns every primitive plane of the result.

  sod_1d              a shock tube of 1000 cells to t = 0.25 through vg_solve, as the scenarios run it; latency
  euler_2d_small      a 2D scenario grid of the size of the reference's own runs: launches and latency
  euler_2d            the 4096^2 four-quadrant Riemann problem, exact FP64 form: the largest grid in earnest use
  euler_2d_mixed      the same in the mixed FP32/FP64 form
  mhd_2d              the 2048^2 periodic MHD vortex from host planes (vg_solve), exact form
  mhd_2d_mixed        the same in the mixed form
  hpr_2d_forcing      1024^2 HPR with the reference's RK4 relaxation source at 13 sub-cycles per half step
  hpr_2d_stiff_mixed  1024^2 HPR with the stiff relaxation source, mixed form (the form users choose at small tau)
  batch_forward       a ragged batch of 4096 1D Riemann problems, 200 to 4000 cells each
  batch_gradient      the discrete adjoint of such a batch with binomial checkpointing
  reduced_2d          the two-material Euler bubble with the volume-fraction reinitialisation
  mhd_reduced_2d      the two-material MHD disc on an odd grid with GLM damping sub-cycles

exact() restates each scheme in plain torch, FP64, one rounding per operation.
"""
import math

import numpy as np
import torch

import vanguard_b200 as vg

CFL = 0.8
LIMITERS = (vg.SUPERBEE, vg.VANLEER, vg.MINBEE)
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


# ------------------------------------------------------------------------------------------------- the cases

def listed():
    return [
        # time to solution of the smallest problem anybody runs
        {"name": "sod_1d", "kind": "euler_1d", "nx": 1000, "t_end": 0.25, "steps": 0, "cfl": 0.9, "limiter": vg.MINBEE},
        # the reference's 2D scenarios have grids of this order: a step is four short launches
        {"name": "euler_2d_small", "kind": "euler_2d", "nx": 130, "ny": 97, "steps": 100, "limiter": vg.SUPERBEE,
         "precision": vg.FP64, "boundary": vg.TRANSMISSIVE},
        # the headline grid, in both forms
        {"name": "euler_2d", "kind": "euler_2d", "nx": 4096, "ny": 4096, "steps": 20, "limiter": vg.SUPERBEE,
         "precision": vg.FP64, "boundary": vg.TRANSMISSIVE},
        {"name": "euler_2d_mixed", "kind": "euler_2d", "nx": 4096, "ny": 4096, "steps": 20, "limiter": vg.SUPERBEE,
         "precision": vg.MIXED, "boundary": vg.TRANSMISSIVE},
        # MHD from host planes, which is what selects the planar variant (w = Bz = 0)
        {"name": "mhd_2d", "kind": "mhd_2d", "nx": 2048, "ny": 2048, "steps": 60, "limiter": vg.SUPERBEE,
         "precision": vg.FP64, "boundary": vg.PERIODIC},
        {"name": "mhd_2d_mixed", "kind": "mhd_2d", "nx": 2048, "ny": 2048, "steps": 60, "limiter": vg.SUPERBEE,
         "precision": vg.MIXED, "boundary": vg.PERIODIC},
        # HPR heat conduction with the reference's explicit source, and with the stiff relaxation
        {"name": "hpr_2d_forcing", "kind": "hpr_2d", "nx": 1024, "ny": 1024, "steps": 2, "limiter": vg.SUPERBEE,
         "precision": vg.FP64, "tau1": 5.1e-4, "tau2": 7.2e-6, "subcycles": 13, "stiff": False},
        {"name": "hpr_2d_stiff_mixed", "kind": "hpr_2d", "nx": 1024, "ny": 1024, "steps": 20, "limiter": vg.SUPERBEE,
         "precision": vg.MIXED, "tau1": 5.1e-4, "tau2": 7.2e-6, "subcycles": 0, "stiff": True},
        # parameter studies: many small problems at once, and the gradient of a misfit through them
        {"name": "batch_forward", "kind": "batch", "ninst": 4096, "nmin": 200, "nmax": 4000, "steps": 200,
         "limiter": vg.SUPERBEE},
        {"name": "batch_gradient", "kind": "gradient", "ninst": 1024, "nmin": 200, "nmax": 4000, "steps": 60,
         "checkpoints": 12, "limiter": vg.SUPERBEE},
        # two materials
        {"name": "reduced_2d", "kind": "reduced_2d", "nx": 2048, "ny": 2048, "steps": 20, "limiter": vg.SUPERBEE,
         "reinit": 10},
        {"name": "mhd_reduced_2d", "kind": "mhd_reduced_2d", "nx": 1001, "ny": 777, "steps": 6, "limiter": vg.VANLEER,
         "subcycles": 1, "reinit": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["euler_1d", "euler_2d", "mhd_2d", "hpr_2d", "batch", "gradient", "reduced_2d", "mhd_reduced_2d"])
    limiter = rng.choice(LIMITERS)
    if kind == "euler_1d":
        nx = _log_int(rng, 100, 200000)
        if nx <= 2000:
            return {"kind": kind, "nx": nx, "t_end": rng.uniform(0.1, 0.25), "steps": 0, "cfl": rng.uniform(0.5, 0.9),
                    "limiter": limiter}
        return {"kind": kind, "nx": nx, "t_end": 0.0, "steps": rng.randint(50, 200), "cfl": rng.uniform(0.5, 0.9),
                "limiter": limiter}
    if kind in ("euler_2d", "mhd_2d"):
        top = 4096 if kind == "euler_2d" else 2048
        return {"kind": kind, "nx": _log_int(rng, 64, top), "ny": _log_int(rng, 64, top), "steps": rng.randint(5, 20),
                "limiter": limiter, "precision": rng.choice([vg.FP64, vg.FP64, vg.MIXED]),
                "boundary": vg.PERIODIC if kind == "mhd_2d" else rng.choice([vg.TRANSMISSIVE, vg.PERIODIC])}
    if kind == "hpr_2d":
        nx, ny = _log_int(rng, 64, 1024), _log_int(rng, 64, 1024)
        stiff = rng.random() < 0.5
        sub = rng.randint(1, 13)
        # the explicit source is stable for sub-steps up to 2.5 tau; the wave speed of this field is at least 2
        tau = 0.5 * (1.5 * CFL / nx / 2.0) / (2.5 * sub)
        return {"kind": kind, "nx": nx, "ny": ny, "steps": 10 if stiff else 2, "limiter": limiter,
                "precision": rng.choice([vg.FP64, vg.MIXED]), "tau1": tau * rng.uniform(1.0, 50.0),
                "tau2": tau * rng.uniform(1.0, 2.0), "subcycles": 0 if stiff else sub, "stiff": stiff}
    if kind in ("batch", "gradient"):
        case = {"kind": kind, "ninst": _log_int(rng, 16, 4096 if kind == "batch" else 1024),
                "nmin": rng.randint(20, 200), "nmax": _log_int(rng, 300, 4000), "steps": rng.randint(10, 60),
                "limiter": limiter}
        if kind == "gradient":
            case["checkpoints"] = rng.randint(4, 16)
        return case
    if kind == "reduced_2d":
        return {"kind": kind, "nx": _log_int(rng, 64, 2048), "ny": _log_int(rng, 64, 2048), "steps": rng.randint(4, 20),
                "limiter": limiter, "reinit": rng.choice([0, 5, 10])}
    return {"kind": kind, "nx": _log_int(rng, 64, 1001), "ny": _log_int(rng, 64, 777), "steps": rng.randint(2, 6),
            "limiter": limiter, "subcycles": rng.randint(0, 1), "reinit": rng.choice([0, 3])}


# ---------------------------------------------------------------------------------------------- their inputs

def _uniform(gen, lo, hi, shape):
    return lo + (hi - lo) * torch.rand(shape, generator=gen, dtype=torch.float64, device=DEVICE)


def _normal(gen, shape):
    return torch.randn(shape, generator=gen, dtype=torch.float64, device=DEVICE)


def _grid(nx, ny):
    x = (torch.arange(nx, dtype=torch.float64, device=DEVICE) + 0.5) / nx
    y = (torch.arange(ny, dtype=torch.float64, device=DEVICE) + 0.5) / ny
    return x[None, :].expand(ny, nx), y[:, None].expand(ny, nx)


def _disc(nx, ny):
    i = torch.arange(ny, dtype=torch.float64, device=DEVICE)[:, None]
    j = torch.arange(nx, dtype=torch.float64, device=DEVICE)[None, :]
    return ((i - 0.5 * ny) ** 2 + (j - 0.5 * nx) ** 2).sqrt() <= 0.2 * nx


def _planes(case, seed):
    """The seeded initial primitive planes of a grid case, (nvar, ny, nx) or (nvar, nx) on the GPU."""
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed))
    kind, nx = case["kind"], case["nx"]
    new = lambda *s: torch.zeros(s, dtype=torch.float64, device=DEVICE)  # noqa: E731
    if kind == "euler_1d":  # a shock tube with left and right states about Sod's
        W = new(6, nx)
        left = torch.arange(nx, device=DEVICE) <= 0.5 * nx
        f = _uniform(gen, 0.8, 1.2, 4)
        W[0] = torch.where(left, 1.0 * f[0], 0.125 * f[1])
        W[4] = torch.where(left, 1.0 * f[2], 0.1 * f[3])
        W[5] = 1.0
        return W
    ny = case["ny"]
    if kind == "euler_2d":  # four quadrants, rho and p ~ U[0.1, 2], u and v ~ U[-1, 1]
        q = 2 * (torch.arange(ny, device=DEVICE) >= ny // 2).long()[:, None] + (torch.arange(nx, device=DEVICE) >= nx // 2).long()
        W = new(6, ny, nx)
        for plane, lo, hi in ((0, 0.1, 2.0), (1, -1.0, 1.0), (2, -1.0, 1.0), (4, 0.1, 2.0)):
            W[plane] = _uniform(gen, lo, hi, 4)[q]
        W[5] = 1.0
        return W
    x, y = _grid(nx, ny)
    two_pi = 2.0 * math.pi
    if kind == "mhd_2d":  # Orszag-Tang-type vortex with seeded noise on the density and pressure
        g = 5.0 / 3.0
        W = new(9, ny, nx)
        W[0] = g * g + 1e-3 * _normal(gen, (ny, nx))
        W[1] = -torch.sin(two_pi * y)
        W[2] = torch.sin(two_pi * x)
        W[4] = g + 1e-3 * _normal(gen, (ny, nx))
        W[5] = -torch.sin(two_pi * y) / math.sqrt(4 * math.pi)
        W[6] = torch.sin(2 * two_pi * x) / math.sqrt(4 * math.pi)
        return W
    if kind == "hpr_2d":  # smooth density wave and seeded velocity phases, A = I, J = 0
        phi = _uniform(gen, 0.0, two_pi, 5)
        W = new(17, ny, nx)
        W[0] = 1.0 + 0.2 * torch.sin(two_pi * (2 * x + y) + phi[0])
        W[1] = 1.0
        W[2] = W[6] = W[10] = 1.0
        W[11] = 0.05 * (torch.sin(two_pi * y + phi[1]) + torch.cos(two_pi * x + phi[2]))
        W[12] = 0.05 * (torch.sin(two_pi * x + phi[3]) + torch.cos(two_pi * y + phi[4]))
        return W
    inside = _disc(nx, ny)
    f = _uniform(gen, 0.9, 1.1, 4)
    if kind == "reduced_2d":  # the bubble of material 1 in material 2
        W = new(7, ny, nx)
        W[0] = torch.where(inside, 0.999, 0.001)
        W[4] = 1.0 * f[0]
        W[5] = 0.125 * f[1]
        W[6] = torch.where(inside, 1.0 * f[2], 0.1 * f[3])
        return W
    W = new(11, ny, nx)  # mhd_reduced_2d: the Brio-Wu states inside and outside of a disc
    W[0] = torch.where(inside, 0.999, 0.001)
    W[4] = 1.0 * f[0]
    W[5] = 0.125 * f[1]
    W[6] = torch.where(inside, 1.0 * f[2], 0.1 * f[3])
    W[7] = 0.75
    W[8] = torch.where(inside, 1.0, -1.0)
    return W


def _batch_inputs(case, seed):
    """(cells, widths, gammas as host arrays, the (6, total) planes on the GPU) of a ragged batch of Riemann problems."""
    k = case["ninst"]  # the sizes belong to the case, the problems on them to the seed
    ncell = np.random.default_rng([k, case["nmin"], case["nmax"]]).integers(case["nmin"], case["nmax"] + 1, k).astype(np.int32)
    rng = np.random.default_rng(seed)
    gamma = rng.uniform(1.2, 1.67, k)
    states = [rng.uniform(lo, hi, k) for lo, hi in ((0.1, 2.0), (-1.0, 1.0), (0.1, 10.0)) * 2]
    inst = torch.from_numpy(np.repeat(np.arange(k), ncell)).to(DEVICE)
    cell = torch.from_numpy(np.concatenate([np.arange(n) for n in ncell])).to(DEVICE)
    left = cell <= 0.5 * torch.from_numpy(ncell).to(DEVICE)[inst]
    s = torch.from_numpy(np.stack(states)).to(DEVICE)
    W = torch.zeros((6, inst.numel()), dtype=torch.float64, device=DEVICE)
    for row, plane in enumerate((0, 1, 4)):
        W[plane] = torch.where(left, s[row][inst], s[row + 3][inst])
    W[5] = 1.0
    return ncell, 1.0 / ncell, gamma, W


def _target(W, seed):
    """The density that the gradient case fits: the initial one with seeded noise."""
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed) + 1)
    return (W[0] * (1.0 + 0.1 * _normal(gen, W[0].shape))).contiguous()


MODELS = {"euler_1d": vg.EULER, "euler_2d": vg.EULER, "mhd_2d": vg.MHD, "hpr_2d": vg.HPR,
          "reduced_2d": vg.EULER_REDUCED, "mhd_reduced_2d": vg.MHD_REDUCED}


def _params(case):
    if case["kind"] in ("euler_1d", "euler_2d"):
        return [1.4, 0.0, 25.0, 0.0, 0.25, 250.0]
    if case["kind"] == "mhd_2d":
        return [5.0 / 3.0, 0.0, 0.0]
    if case["kind"] == "hpr_2d":  # gamma, p_inf, c_v, rho0, T0, c_s, alpha, tau1, tau2, T_ref, p_ref, thermal
        return [1.4, 0.0, 2.5, 1.0, 1.0, 1.0, 1.0, case["tau1"], case["tau2"], 0.0, 1.0, 1.0]
    return [1.4, 0.0, 1.67, 0.0]


def _pinned(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=torch.cuda.is_available())
    out.copy_(t)
    return out


def prepare(case, seed):
    if case["kind"] in ("batch", "gradient"):
        ncell, dx, gamma, W = _batch_inputs(case, seed)
        state = {"case": case, "W": W, "batch": vg.Batch(ncell, dx, gamma)}
        if case["kind"] == "batch":
            state["out"] = torch.empty(W.shape, dtype=W.dtype, pin_memory=torch.cuda.is_available())
        else:
            state["target"] = _target(W, seed)
            state["grad"] = (torch.empty_like(W), torch.empty(case["ninst"], dtype=W.dtype, device=DEVICE))
        return state
    W = _planes(case, seed)
    solver = vg.Solver(MODELS[case["kind"]], case["nx"], case.get("ny", 1), _params(case),
                       precision=case.get("precision", vg.FP64), boundary=case.get("boundary", vg.TRANSMISSIVE))
    if case["kind"] in ("euler_1d", "mhd_2d"):  # these take host planes: their compact variants are chosen from them
        W = _pinned(W)
        return {"case": case, "solver": solver, "W": W, "out": torch.empty(W.shape, dtype=W.dtype, pin_memory=W.is_pinned())}
    return {"case": case, "solver": solver, "W": W, "out": torch.empty_like(W)}


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.upload(state["W"])
        dt = b.run(CFL, case["steps"], limiter=case["limiter"])
        b.download(out=state["out"].numpy())
        return {"planes": state["out"], "dt": dt}
    if case["kind"] == "gradient":
        b = state["batch"]
        b.upload(state["W"])
        loss, g, gg, _, _ = b.gradient(state["target"], CFL, case["steps"], limiter=case["limiter"],
                                       checkpoints=case["checkpoints"], out=state["grad"])
        return {"loss": loss, "planes": g, "gamma": gg}
    s, dx = state["solver"], 1.0 / case["nx"]
    if case["kind"] in ("euler_1d", "mhd_2d"):
        _, t, it = s.solve(state["W"].numpy(), dx, case.get("cfl", CFL), t_end=case.get("t_end", 0.0), steps=case["steps"],
                           limiter=case["limiter"], out=state["out"].numpy())
    else:
        s.upload(state["W"])
        t, it = s.run(dx, CFL, steps=case["steps"], limiter=case["limiter"], subcycles=case.get("subcycles", 0),
                      stiff=case.get("stiff", False), reinit=case.get("reinit", 0))
        s.download(out=state["out"])
    return {"planes": state["out"], "t": t, "steps": it}


# planes that a state carries and operations of one cell in one sweep (or one source sub-cycle), counted from the
# scheme: slopes, half-step evolution, three fluxes, conversions and update; a division or square root is one
CARRIED = {"euler_1d": 3, "euler_2d": 4, "mhd_2d": 7, "hpr_2d": 17, "reduced_2d": 6, "mhd_reduced_2d": 11}
SWEEP_FLOPS = {"euler_1d": 220, "euler_2d": 300, "mhd_2d": 560, "hpr_2d": 2600, "reduced_2d": 600, "mhd_reduced_2d": 1100}
SOURCE_FLOPS = {"hpr_2d": 13000, "mhd_reduced_2d": 6000}
RELAX_FLOPS = 1500


def work(case):
    steps = case["steps"]
    if case["kind"] in ("batch", "gradient"):
        cells = case["ninst"] * 0.5 * (case["nmin"] + case["nmax"])
        if case["kind"] == "batch":
            return {"bytes": 2 * 3 * 8 * cells, "flops": SWEEP_FLOPS["euler_1d"] * cells * steps}
        # the state and the target in, the gradient out; forward and reverse of every step
        return {"bytes": (3 + 1 + 3) * 8 * cells, "flops": 3 * SWEEP_FLOPS["euler_1d"] * cells * steps}
    kind = case["kind"]
    cells = case["nx"] * case.get("ny", 1)
    if not steps:  # time-driven: the fastest wave of these tubes is about 2.2
        steps = max(1, int(case["t_end"] * 2.2 * case["nx"] / case["cfl"]))
    flops = SWEEP_FLOPS[kind] * (1 if kind == "euler_1d" else 3)
    flops += 2 * case.get("subcycles", 0) * SOURCE_FLOPS.get(kind, 0)
    flops += 2 * RELAX_FLOPS if case.get("stiff") else 0
    return {"bytes": 2 * 8 * CARRIED[kind] * cells, "flops": flops * cells * steps}


# ----------------------------------------------------------- the same schemes in plain torch, FP64 throughout
# States are lists of component tensors.  Each model gives the conserved vector of its primitives and back, the
# flux along an axis, the wave speed, the default-constructed state and, where it has one, the source.

def _sq(*v):
    s = v[0] * v[0]
    for x in v[1:]:
        s = s + x * x
    return s


class _Euler:
    """rho, u, v, p | rho, rho u, rho v, rho E; g may be a tensor (one gamma per instance of a batch)."""

    planes, constant = (0, 1, 2, 4), {5: 1.0}
    default = (1.0, 0.0, 0.0, 1.0)

    def __init__(self, g):
        self.g = g

    def cons(self, W):
        r, u, v, p = W
        return [r, r * u, r * v, r * (0.5 * _sq(u, v) + p / ((self.g - 1) * r))]

    def _parts(self, U):
        r = U[0]
        u, v, E = U[1] / r, U[2] / r, U[3] / r
        return r, u, v, E, ((E - 0.5 * _sq(u, v)) * (self.g - 1)) * r

    def prim(self, U, keep=None):
        r, u, v, _, p = self._parts(U)
        return [r, u, v, p]

    def flux(self, U, axis):
        r, u, v, E, p = self._parts(U)
        n = u if axis == 0 else v
        F = [r * n, r * (n * u), r * (n * v), r * (n * E) + n * p]
        F[1 + axis] = F[1 + axis] + p
        return F

    def wave(self, W, dims):
        c = ((self.g * W[3]) / W[0]).sqrt()
        return (W[1].abs() if dims == 1 else torch.maximum(W[1].abs(), W[2].abs())) + c


class _MHD:
    """rho, u, v, w, p, B, psi | rho, m, E, B, psi with the GLM speed ch of the step."""

    planes, constant = tuple(range(9)), {}
    default = (1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 0.0)

    def __init__(self, g):
        self.g, self.ch = g, 0.0

    def cons(self, W):
        r, u, v, w, p, bx, by, bz, psi = W
        E = r * (0.5 * _sq(u, v, w) + p / ((self.g - 1) * r)) + 0.5 * _sq(bx, by, bz)
        return [r, r * u, r * v, r * w, E, bx, by, bz, psi]

    def _parts(self, U):
        r = U[0]
        vel = [U[k] / r for k in (1, 2, 3)]
        b2 = _sq(*U[5:8])
        e = (U[4] - 0.5 * b2) / r - 0.5 * _sq(*vel)
        return r, vel, b2, (e * (self.g - 1)) * r

    def prim(self, U, keep=None):
        r, vel, _, p = self._parts(U)
        return [r, *vel, p, *U[5:]]

    def flux(self, U, axis):
        r, vel, b2, p = self._parts(U)
        B, psi, E = U[5:8], U[8], U[4]
        n, bn = vel[axis], B[axis]
        vb = (vel[0] * B[0] + vel[1] * B[1]) + vel[2] * B[2]
        mom = [r * (n * vel[k]) - bn * B[k] for k in range(3)]
        mom[axis] = ((r * (n * n) + p) + 0.5 * b2) - bn * bn
        F = [r * n, *mom, ((E + p) + 0.5 * b2) * n - vb * bn]
        F += [psi if k == axis else B[k] * n - bn * vel[k] for k in range(3)]
        return F + [(self.ch * self.ch) * bn]

    def _fast(self, W, bn):
        r = W[0]
        c = ((self.g * W[4]) / r).sqrt()
        a = _sq(*W[5:8]).sqrt() / r.sqrt()
        s = c * c + a * a
        return (0.5 * (s + (s * s - 4.0 * ((c * c) * (bn * bn) / r)).sqrt())).sqrt()

    def wave(self, W, dims):
        return torch.maximum(W[1].abs(), W[2].abs()) + torch.maximum(self._fast(W, W[5]), self._fast(W, W[6]))


def _clamp(a):
    return a.clamp(0.001, 0.999)


class _Reduced:
    """alpha1, u, v, rho1, rho2, p | rho, rho alpha1, rho u, rho v, alpha1 rho1, alpha2 rho2, rho E."""

    planes, constant = (0, 1, 2, 4, 5, 6), {}
    default = (0.999, 0.0, 0.0, 1.0, 1.0, 1.0)
    densities = (3, 4)

    def __init__(self, g1, g2):
        self.g1, self.g2 = g1, g2

    def cons(self, W):
        a1 = _clamp(W[0])
        a2 = 1.0 - a1
        _, u, v, r1, r2, p = W
        r = a1 * r1 + a2 * r2
        k = 0.5 * _sq(u, v)
        E1, E2 = p / ((self.g1 - 1) * r) + k, p / ((self.g2 - 1) * r) + k
        return [r, r * a1, r * u, r * v, a1 * r1, a2 * r2, r * (a1 * E1 + a2 * E2)]

    def _parts(self, U):
        r = U[0]
        a1 = _clamp(U[1] / r)
        a2 = 1.0 - a1
        u, v, E = U[2] / r, U[3] / r, U[6] / r
        e = E - 0.5 * _sq(u, v)
        p = a1 * ((e * (self.g1 - 1)) * r) + a2 * ((e * (self.g2 - 1)) * r)
        return r, a1, a2, u, v, U[4] / a1, U[5] / a2, E, p

    def prim(self, U, keep=None):
        _, a1, _, u, v, r1, r2, _, p = self._parts(U)
        return [a1, u, v, r1, r2, p]

    def flux(self, U, axis):
        r, a1, a2, u, v, r1, r2, E, p = self._parts(U)
        n = u if axis == 0 else v
        F = [r * n, r * (n * a1), r * (n * u), r * (n * v), a1 * (r1 * n), a2 * (r2 * n), r * (n * E) + n * p]
        F[2 + axis] = F[2 + axis] + p
        return F

    def wave(self, W, dims):
        c = torch.maximum(((self.g1 * W[5]) / W[3]).sqrt(), ((self.g2 * W[5]) / W[4]).sqrt())
        return torch.maximum(W[1].abs(), W[2].abs()) + c


class _MHDReduced:
    """alpha1, u, v, w, rho1, rho2, p, B, psi; both materials' fast speeds take material 2's density."""

    planes, constant = tuple(range(11)), {}
    default = (0.999, 0.0, 0.0, 0.0, 1.0, 1.0, 1.0, 0.0, 0.0, 0.0, 0.0)
    densities = (4, 5)

    def __init__(self, g1, g2):
        self.g1, self.g2, self.ch = g1, g2, 0.0

    def cons(self, W):
        a1 = _clamp(W[0])
        a2 = 1.0 - a1
        u, v, w, r1, r2, p = W[1:7]
        B = W[7:10]
        r = a1 * r1 + a2 * r2
        k, m = 0.5 * _sq(u, v, w), 0.5 * _sq(*B)
        h1, h2 = r * (k + p / ((self.g1 - 1) * r)), r * (k + p / ((self.g2 - 1) * r))
        return [r, r * a1, r * u, r * v, r * w, a1 * r1, a2 * r2, a1 * (h1 + m) + a2 * (h2 + m), *B, W[10]]

    def _parts(self, U):
        r = U[0]
        a1 = _clamp(U[1] / r)
        a2 = 1.0 - a1
        vel = [U[k] / r for k in (2, 3, 4)]
        b2 = _sq(*U[8:11])
        e = (U[7] - 0.5 * b2) / r - 0.5 * _sq(*vel)
        p = a1 * ((e * (self.g1 - 1)) * r) + a2 * ((e * (self.g2 - 1)) * r)
        return r, a1, a2, vel, U[5] / a1, U[6] / a2, b2, p

    def prim(self, U, keep=None):
        _, a1, _, vel, r1, r2, _, p = self._parts(U)
        return [a1, *vel, r1, r2, p, *U[8:]]

    def flux(self, U, axis):
        r, a1, a2, vel, r1, r2, b2, p = self._parts(U)
        B, psi, E = U[8:11], U[11], U[7]
        n, bn = vel[axis], B[axis]
        vb = (vel[0] * B[0] + vel[1] * B[1]) + vel[2] * B[2]
        ch2 = self.ch * self.ch
        mom = [r * (n * vel[k]) - bn * B[k] for k in range(3)]
        mom[axis] = ((r * (n * n) + p) + 0.5 * b2) - bn * bn
        F = [r * n, r * (n * a1), *mom, a1 * (r1 * n), a2 * (r2 * n), ((E + p) + 0.5 * b2) * n - vb * bn]
        F += [psi if k == axis else B[k] * n - bn * vel[k] for k in range(3)]
        return F + [(a1 * ch2 + a2 * ch2) * bn]

    def source(self, U):
        a1 = _clamp(U[1] / U[0])
        a2 = 1.0 - a1
        cp = math.sqrt(self.ch * 0.18)
        ch2, cp2 = self.ch * self.ch, cp * cp
        S = [torch.zeros_like(U[0]) for _ in U]
        S[11] = -((a1 * ch2 + a2 * ch2) / (a1 * cp2 + a2 * cp2)) * U[11]
        return S

    def wave(self, W, dims):
        r, p, B = W[5], W[6], W[7:10]
        a = _sq(*B).sqrt() / r.sqrt()
        best = None
        for g in (self.g1, self.g2):
            c = ((g * p) / r).sqrt()
            s = c * c + a * a
            for bn in B[:2]:
                f = (0.5 * (s + (s * s - 4.0 * ((c * c) * (bn * bn) / r)).sqrt())).sqrt()
                best = f if best is None else torch.maximum(best, f)
        return torch.maximum(W[1].abs(), W[2].abs()) + best


class _HPR:
    """rho, p, A (9), u, v, w, J | rho, rho E, A, rho u, rho v, rho w, rho J: a thermal ideal gas with c_s = alpha =
    rho0 = T0 = 1 and c_v = 2.5."""

    planes, constant = tuple(range(17)), {}
    default = (1.0, 1.0, 1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0)
    cv = 2.5

    def __init__(self, g, tau1, tau2):
        self.g, self.tau1, self.tau2 = g, tau1, tau2

    @staticmethod
    def _mat(A):
        return [[A[3 * i + j] for j in range(3)] for i in range(3)]

    @staticmethod
    def _tmul(a, b):
        return [[(a[0][i] * b[0][j] + a[1][i] * b[1][j]) + a[2][i] * b[2][j] for j in range(3)] for i in range(3)]

    @staticmethod
    def _mul(a, b):
        return [[(a[i][0] * b[0][j] + a[i][1] * b[1][j]) + a[i][2] * b[2][j] for j in range(3)] for i in range(3)]

    @staticmethod
    def _dev(g):
        c = ((g[0][0] + g[1][1]) + g[2][2]) / 3.0
        return [[g[i][j] - c if i == j else g[i][j] for j in range(3)] for i in range(3)]

    def _meso(self, A, J):
        D = self._dev(self._tmul(A, A))
        s = (_sq(*D[0]) + _sq(*D[1])) + _sq(*D[2])
        return 0.25 * s, 0.5 * _sq(*J)

    def cons(self, W):
        r, p, A, vel, J = W[0], W[1], self._mat(W[2:11]), W[11:14], W[14:17]
        dist, heat = self._meso(A, J)
        E = ((p / (r * (self.g - 1.0)) + dist) + 0.5 * _sq(*vel)) + heat
        return [r, r * E, *W[2:11], *[r * x for x in vel], *[r * x for x in J]]

    def _parts(self, U):
        r = U[0]
        A = self._mat(U[2:11])
        vel, J, E = [U[k] / r for k in (11, 12, 13)], [U[k] / r for k in (14, 15, 16)], U[1] / r
        dist, heat = self._meso(A, J)
        e = (E - (0.5 * _sq(*vel) + dist)) - heat
        return r, A, vel, J, E, (e * r) * (self.g - 1.0)

    def _temperature(self, r, p):
        return p / ((r * (self.g - 1.0)) * self.cv)

    def prim(self, U, keep=None):
        r, _, vel, J, _, p = self._parts(U)
        return [r, p, *U[2:11], *vel, *J]

    def flux(self, U, axis):
        r, A, vel, J, E, p = self._parts(U)
        sig = [-r * x for x in self._tmul(A, self._mul(A, self._dev(self._tmul(A, A))))[axis]]
        n, T = vel[axis], self._temperature(r, p)
        F = [r * n, (r * (n * E) + p * n) - ((sig[0] * vel[0] + sig[1] * vel[1]) + sig[2] * vel[2]) + T * J[axis]]
        F += [torch.zeros_like(r) for _ in range(9)]
        for i in range(3):
            F[2 + 3 * i + axis] = (A[i][0] * vel[0] + A[i][1] * vel[1]) + A[i][2] * vel[2]
        for k in range(3):
            m = r * (n * vel[k])
            F.append((m + p if k == axis else m) - sig[k])
        for k in range(3):
            h = r * (n * J[k])
            F.append(h + T if k == axis else h)
        return F

    def source(self, U):
        r, A, vel, J, E, p = self._parts(U)
        d = self._mul(A, self._dev(self._tmul(A, A)))
        det = (A[0][0] * (A[1][1] * A[2][2] - A[2][1] * A[1][2]) - A[0][1] * (A[1][0] * A[2][2] - A[1][2] * A[2][0])) \
            + A[0][2] * (A[1][0] * A[2][1] - A[1][1] * A[2][0])
        th1 = 3.0 * (det ** (5.0 / 3.0) / self.tau1)
        S = [torch.zeros_like(r), torch.zeros_like(r)] + [-d[i][j] * th1 for i in range(3) for j in range(3)]
        th2 = 1.0 / (self.tau2 * (r * (1.0 / self._temperature(r, p))))
        return S + [torch.zeros_like(r) for _ in range(3)] + [(-r * th2) * x for x in J]

    def _speed(self, W, d):
        r, p, A = W[0], W[1], self._mat(W[2:11])
        zero = torch.zeros_like(r)
        G = self._tmul(A, A)
        D = self._dev(G)
        AD = self._mul(A, D)
        Pm = self._tmul(A, AD)
        ir, gm1 = 1.0 / r, self.g - 1.0
        c1, c2 = [[zero] * 5 for _ in range(4)], [[zero] * 4 for _ in range(5)]
        c1[0][1] = ir
        for i in range(3):
            for j in range(3):
                t = (G[d][i] * A[j][d] + G[d][d] * A[j][i]) - (2.0 / 3.0) * (G[d][i] * A[j][d]) + AD[j][i]
                if i == d:
                    t = t + AD[j][d]
                c1[i][2 + j] = -ir * (-r * t)
            c1[i][0] = ir * Pm[d][i]
        dTdp = (1.0 / (r * gm1)) / self.cv
        dTdr = -(gm1 * p) / (((r * gm1) * (r * gm1)) / self.cv)
        c1[3][0], c1[3][1] = dTdr / r, dTdp / r
        dedr = -((gm1 * p) / ((r * gm1) * (r * gm1)))
        cad = ((p / (r * r) - dedr) / (1.0 / (r * gm1))).sqrt()
        c2[0][0] = r
        c2[1][d] = r * (cad * cad)
        for i in range(3):
            c2[1][i] = c2[1][i] + (-r * Pm[d][i] - r * (-Pm[d][i]))
            for j in range(3):
                c2[2 + i][j] = A[i][j]
        ch = (self._temperature(r, p) / self.cv).sqrt() / r
        c2[1][3] = r * ((ch * ch) / dTdp)
        om = [[sum((c1[i][k] * c2[k][j] for k in range(5)), zero) for j in range(4)] for i in range(4)]
        x = [torch.ones_like(r) for _ in range(4)]
        for it in range(11):
            y = [((om[i][0] * x[0] + om[i][1] * x[1]) + om[i][2] * x[2]) + om[i][3] * x[3] for i in range(4)]
            norm = _sq(*y).sqrt()
            if it < 10:
                x = [(1.0 / norm) * v for v in y]
        return norm.sqrt()

    def wave(self, W, dims):
        return torch.maximum(W[11].abs(), W[12].abs()) + torch.maximum(self._speed(W, 0), self._speed(W, 1))


def _slope(uL, u, uR, limiter):
    """The limited slope of one component; the limiter's operand keeps to 1e-5 where a difference is smaller."""
    dm, dp = u - uL, uR - u
    floor = 10.0 ** -5.0
    r = torch.where(dm.abs() < floor, floor, dm) / torch.where(dp.abs() < floor, floor, dp)
    xi = 2.0 / (1.0 + torch.where(r < 0, 1.0, r))
    if limiter == vg.SUPERBEE:
        big = torch.where(xi < r, xi, r)
        big = torch.where(big > 2.0, 2.0, big)
        phi = torch.where(r < 0, 0.0, torch.where(r < 0.5, 2.0 * r, torch.where(r < 1.0, 1.0, big)))
    elif limiter == vg.VANLEER:
        lim = (2.0 * r) / (1.0 + torch.where(r < 0, 1.0, r))
        phi = torch.where(r < 0, 0.0, torch.where(xi < lim, xi, lim))
    else:
        phi = torch.where(r < 0, 0.0, torch.where(r < 1.0, r, torch.where(xi < 1.0, xi, 1.0)))
    return (0.5 * dm + 0.5 * dp) * phi


def _take(state, dim, start, count):
    return [x.narrow(dim, start, count) for x in state]


def _ghosts(W, dim, width, periodic):
    n = W[0].shape[dim]
    k = torch.arange(-width, n + width, device=W[0].device)
    if periodic:
        k = k % n
    elif width == 1:
        k = k.clamp(0, n - 1)
    else:
        k = torch.where(k < 0, -1 - k, torch.where(k >= n, 2 * n - 1 - k, k))
    return [x.index_select(dim, k) for x in W]


def _edges(M, uL, u, uR, axis, half_r, limiter):
    s = [0.5 * _slope(a, b, c, limiter) for a, b, c in zip(uL, u, uR)]
    xl, xr = [a - b for a, b in zip(u, s)], [a + b for a, b in zip(u, s)]
    ev = [half_r * (f - g) for f, g in zip(M.flux(xl, axis), M.flux(xr, axis))]
    return [M.cons(M.prim([a + e for a, e in zip(x, ev)])) for x in (xl, xr)]


def _advance(M, Up, axis, dim, r, rinv, half_r, limiter):
    """New conserved vectors from conserved vectors with two ghost cells a side."""
    n = Up[0].shape[dim] - 4
    a, b = _edges(M, _take(Up, dim, 0, n + 2), _take(Up, dim, 1, n + 2), _take(Up, dim, 2, n + 2), axis, half_r, limiter)
    ua, ub = _take(b, dim, 0, n + 1), _take(a, dim, 1, n + 1)
    fa, fb = M.flux(ua, axis), M.flux(ub, axis)
    ri = M.flux([0.5 * ((x + y) + r * (f - g)) for x, y, f, g in zip(ua, ub, fa, fb)], axis)
    F = [0.5 * (0.5 * ((f + g) + rinv * (x - y)) + h) for x, y, f, g, h in zip(ua, ub, fa, fb, ri)]
    return [u + r * (f.narrow(dim, 0, n) - f.narrow(dim, 1, n)) for u, f in zip(_take(Up, dim, 2, n), F)]


def _sweep(M, W, axis, dt, dx, limiter, periodic):
    dim = W[0].dim() - 1 - axis
    U = M.cons(_ghosts(W, dim, 2, periodic))
    return M.prim(_advance(M, U, axis, dim, dt / dx, dx / dt, 0.5 * (dt / dx), limiter), W)


def _forcing(M, W, dt, dx, limiter, periodic):
    """One RK4 source sub-step with the fractional-flux predictors X(f/2) Y(f) X(f/2)."""
    rest = M.cons(M.prim(M.cons(W)))
    near = {axis: [_take(g, 1 - axis, 0, W[0].shape[1 - axis]) if k == 0 else _take(g, 1 - axis, 2, W[0].shape[1 - axis])
                   for g in [_ghosts(rest, 1 - axis, 1, periodic)] for k in (0, 1)] for axis in (0, 1)}
    U = M.cons(W)
    k = [[dt * s for s in M.source(U)]]
    for stage, f in enumerate((0.5, 0.5, 1.0)):
        Ws = M.prim([u + (0.5 * x if stage < 2 else x) for u, x in zip(U, k[stage])])
        for axis, part in ((0, 0.5 * f), (1, f), (0, 0.5 * f)):
            um = M.cons(Ws)
            s = [0.5 * _slope(a, b, c, limiter) for a, b, c in zip(near[axis][0], um, near[axis][1])]
            fl = M.flux([a - b for a, b in zip(um, s)], axis)
            fr = M.flux([a + b for a, b in zip(um, s)], axis)
            c = part * (dt / dx)
            Ws = M.prim([u + c * (a - b) for u, a, b in zip(um, fl, fr)])
        k.append([dt * s for s in M.source(M.cons(Ws))])
    return M.prim([u + (1.0 / 6.0) * (a + (2.0 * b + (2.0 * c + d))) for u, a, b, c, d in zip(U, *k)], W)


def _reinitialise(M, W):
    """The volume fraction reset about every crossing of 0.5, rows first, then columns; descending crossings first."""
    for dim in (1, 0):
        P = [x if dim == 1 else x.t().contiguous() for x in W]
        lines, n = P[0].shape
        alpha, r1, r2 = P[0].clone(), P[M.densities[0]].clone(), P[M.densities[1]].clone()
        now, before = alpha[:, 1:], alpha[:, :-1]
        found = [((now < 0.5) & (before >= 0.5), 0.999, 0.001), ((now > 0.5) & (before <= 0.5), 0.001, 0.999)]
        for mask, low, high in found:
            count = mask.sum(1)
            rank = mask.cumsum(1)
            for k in range(1, min(100, int(count.max())) + 1):
                line = torch.nonzero(count >= k).flatten()
                at = ((rank == k) & mask)[line].int().argmax(1) + 1
                for off in (-2, -1, 0, 1):
                    j = at + off
                    ok = (j >= 0) & (j < n)
                    i, jj = line[ok], j[ok]
                    a = alpha[i, jj]
                    r = a * r1[i, jj] + (1.0 - a) * r2[i, jj]
                    r1[i, jj] = r
                    r2[i, jj] = r
                    alpha[i, jj] = low if off < 0 else high
        P[0], P[M.densities[0]], P[M.densities[1]] = alpha, r1, r2
        W = [x if dim == 1 else x.t().contiguous() for x in P]
    return W


def _model(case):
    kind = case["kind"]
    if kind in ("euler_1d", "euler_2d"):
        return _Euler(1.4)
    if kind == "mhd_2d":
        return _MHD(5.0 / 3.0)
    if kind == "hpr_2d":
        return _HPR(1.4, case["tau1"], case["tau2"])
    return (_Reduced if kind == "reduced_2d" else _MHDReduced)(1.4, 1.67)


def _first_at(x, top):
    """The index along dim 1 of the first element that equals the row's maximum."""
    return (x == top).int().argmax(1)


def _batch_exact(case, seed):
    """All instances as the rows of one padded array; the gradient by reverse differentiation of the same steps."""
    ncell, dx, gamma, planes = _batch_inputs(case, seed)
    n = torch.from_numpy(ncell.astype(np.int64)).to(planes.device)
    width, k = int(ncell.max()), case["ninst"]
    off = torch.cumsum(n, 0) - n
    col = torch.arange(width, device=planes.device)
    inside = col[None, :] < n[:, None]
    at = off[:, None] + torch.minimum(col[None, :], n[:, None] - 1)
    cells = torch.arange(-2, width + 2, device=planes.device)[None, :].expand(k, -1)
    end = n[:, None]
    ghost = torch.where(cells < 0, -1 - cells, torch.where(cells >= end, 2 * end - 1 - cells, cells)).clamp(0, width - 1)
    dx = torch.from_numpy(dx).to(planes.device)
    grad = case["kind"] == "gradient"
    g = torch.from_numpy(gamma).to(planes.device).requires_grad_(grad)
    W0 = planes.clone().requires_grad_(grad)
    W = [W0[p][at] for p in (0, 1, 4)]
    last = [None]

    def step(r0, u0, p0, g, scale):
        M = _Euler(g[:, None])
        W = [r0, u0, torch.zeros_like(r0), p0]
        s = torch.where(inside, M.wave(W, 1), -1.0)
        top = s.gather(1, _first_at(s.detach(), s.detach().amax(1, keepdim=True))[:, None])[:, 0]
        dt = CFL * (dx / top)
        if scale:
            dt = dt * 0.2
        last[0] = dt.detach()
        r, rinv = (dt / dx)[:, None], (dx / dt)[:, None]
        U = M.cons([x.gather(1, ghost) for x in W])
        out = M.prim(_advance(M, U, 0, 1, r, rinv, 0.5 * r, case["limiter"]))
        return [torch.where(inside, out[j], W[j]) for j in (0, 1, 3)]

    from torch.utils.checkpoint import checkpoint
    for i in range(case["steps"]):
        W = checkpoint(step, *W, g, i <= 5, use_reentrant=False) if grad else step(*W, g, i <= 5)
    if not grad:
        out = torch.zeros_like(planes)
        for p, x in zip((0, 1, 4), W):
            out[p] = x[inside]
        out[5] = 1.0
        return {"planes": out, "dt": last[0]}
    loss = ((W[0][inside] - _target(planes, seed)) ** 2).sum()
    loss.backward()
    return {"loss": float(loss), "planes": W0.grad, "gamma": g.grad}


def exact(case, seed):
    if case["kind"] in ("batch", "gradient"):
        return _batch_exact(case, seed)
    if case.get("stiff"):
        return None  # an eigen-decomposition of every cell twice a step: over a minute
    M = _model(case)
    planes = _planes(case, seed)
    if planes.dim() == 2:
        planes = planes[:, None, :]
    W = [planes[p] for p in M.planes]
    dims = 1 if case["kind"] == "euler_1d" else 2
    dx, cfl, limiter = 1.0 / case["nx"], case.get("cfl", CFL), case["limiter"]
    periodic = case.get("boundary", vg.TRANSMISSIVE) == vg.PERIODIC
    corner = [torch.full((1, 1), v, dtype=torch.float64, device=planes.device) for v in M.default]
    t, it, t_end = 0.0, 0, case.get("t_end", 0.0)
    while (t < t_end) if t_end > 0.0 else (it < case["steps"]):
        top = float(M.wave(W, dims).max())
        if dims == 2:  # the padded grid's corners hold default-constructed cells
            top = max(top, float(M.wave(corner, dims).max()))
        dt = cfl * (dx / top) * (0.2 if it <= 5 else 1.0)
        if t_end > 0.0 and t + dt > t_end:
            dt = t_end - t
        M.ch = top
        sub = case.get("subcycles", 0)
        for _ in range(sub):
            W = _forcing(M, W, 0.5 * (dt / sub), dx, limiter, periodic)
        for axis, part in ((0, dt),) if dims == 1 else ((0, dt * 0.5), (1, dt), (0, dt * 0.5)):
            W = _sweep(M, W, axis, part, dx, limiter, periodic)
        for _ in range(sub):
            W = _forcing(M, W, 0.5 * (dt / sub), dx, limiter, periodic)
        t, it = t + dt, it + 1
        if case.get("reinit", 0) and it % case["reinit"] == 0:
            W = _reinitialise(M, W)
    out = torch.zeros_like(planes)
    for p, x in zip(M.planes, W):
        out[p] = x
    for p, v in M.constant.items():
        out[p] = v
    return {"planes": out[:, 0] if dims == 1 else out, "t": t, "steps": it}
