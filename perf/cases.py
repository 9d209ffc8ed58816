"""Timed cases of the evolution path: what each one stands for, its inputs, one
pass through `Evolution`, the work the pass cannot do without, and the same
pass in plain 64-bit torch.

A case is one context of periodic boxes ("boxes": "NXxNYxNZ" texts joined by
commas) of one matter model, stencil order, precision and lapse.  A pass is
either `steps` RK4 steps (`what` = "step"; the outputs are the new `_p`
registers, the device buffers the context owns) or one constraint evaluation of
the current state (`what` = "constraints", which a run does at its output
steps).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from cosmograph_b200.evolution import BoxConfig, Evolution
from cosmograph_b200.state import BoxState

RHO = 3.0 / math.pi / 8.0  # the density of H = 1
LAMBDA = 1.0e-6 * RHO
MASS = 1.0
MATTER = {"vacuum": 0, "dust": 1, "scalar": 2}
NFIELDS = {"vacuum": 18, "dust": 22, "scalar": 23}
SYM = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
PAIRS = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))
G, PHI, A, K, GAM, ALPHA, MAT = 0, 6, 7, 13, 14, 17, 18


def _case(name, what, boxes, matter, order, precision, steps, lapse="Harmonic", ko=0.0, z4c=False):
    c = {"what": what, "boxes": boxes, "matter": matter, "order": order, "precision": precision, "steps": steps,
         "lapse": lapse, "ko": ko, "z4c": z4c}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest box of the shipped configurations: latency and launches count; ten steps between two looks
        _case("dust_32_o4_fp64", "step", "32x32x32", "dust", 4, "fp64", 10),
        # the development box: one 64^3 box at order 4
        _case("dust_64_o4_fp64", "step", "64x64x64", "dust", 4, "fp64", 4),
        # the headline box, in the parity arithmetic and in the FP32-mixed form
        _case("dust_256_o8_fp64", "step", "256x256x256", "dust", 8, "fp64", 1),
        _case("dust_256_o8_mixed", "step", "256x256x256", "dust", 8, "mixed", 1),
        # FMA contraction, a box of ordinary size
        _case("dust_128_o8_fma", "step", "128x128x128", "dust", 8, "fp64_fma", 2),
        # scalar-field matter; 1/192 is no power of two
        _case("scalar_192_o8_fp64", "step", "192x192x192", "scalar", 8, "fp64", 1),
        _case("scalar_128_o8_mixed", "step", "128x128x128", "scalar", 8, "mixed", 2),
        # an ensemble of uneven boxes advanced together
        _case("ensemble_o4_mixed", "step", "32x32x32,32x32x32,64x64x64,64x64x64,96x96x96,96x96x96", "dust", 4, "mixed",
              2),
        # boxes of unequal odd sides: ragged bricks, no aligned rows
        _case("dust_ragged_o6_fp64", "step", "101x85x67", "dust", 6, "fp64", 2),
        _case("dust_ragged_o8_mixed", "step", "110x98x90", "dust", 8, "mixed", 2),
        # the physics options together: Z4c damping, dissipation, a lapse with the grid average of K
        _case("vacuum_z4c_96_o8_fp64", "step", "96x96x96", "vacuum", 8, "fp64", 2, "OnePlusLog", 0.1, True),
        # an output step: the constraint statistics of the current state
        _case("constraints_128_o8", "constraints", "128x128x128", "dust", 8, "fp64", 1),
    ]


def draw(rng):
    def side():
        return int(round(math.exp(rng.uniform(math.log(24.0), math.log(160.0)))))

    matter = rng.choice(["dust", "dust", "scalar", "vacuum"])
    precision = rng.choice(["fp64", "mixed", "mixed", "fp64", "fp64_fma"])
    order = rng.choice([2, 4, 6, 8, 8])
    lapse = rng.choice(["Harmonic", "Harmonic", "OnePlusLog"])
    ko = 0.1 if order in (2, 8) and rng.random() < 0.25 else 0.0
    z4c = matter == "vacuum" and precision != "mixed" and rng.random() < 0.5
    what = "constraints" if rng.random() < 0.1 else "step"
    boxes = ["%dx%dx%d" % (side(), side(), side())]
    if what == "step" and rng.random() < 0.25:
        boxes += ["%dx%dx%d" % (side(), side(), side()) for _ in range(rng.randint(1, 5))]
    return _case(None, what, ",".join(boxes), matter, order, precision, rng.randint(1, 3) if what == "step" else 1,
                 lapse, ko, z4c)


def _shapes(case):
    return [tuple(int(s) for s in b.split("x")) for b in case["boxes"].split(",")]


def _spacing(shape):
    dx = 1.0 / shape[0]
    return dx, 0.1 * dx


# ---------------------------------------------------------------------------
# centred differences of order 2, 4, 6, 8 on periodic torch grids
# ---------------------------------------------------------------------------
D1 = {2: (1 / 2,), 4: (2 / 3, -1 / 12), 6: (3 / 4, -3 / 20, 1 / 60), 8: (4 / 5, -1 / 5, 4 / 105, -1 / 280)}
D2 = {2: (-2.0, 1.0), 4: (-5 / 2, 4 / 3, -1 / 12), 6: (-49 / 18, 3 / 2, -3 / 20, 1 / 90),
      8: (-205 / 72, 8 / 5, -1 / 5, 8 / 315, -1 / 560)}
DM = {2: (1 / 4,), 4: (1 / 3, -1 / 48), 6: (135 / 360, -13.5 / 360, 1 / 360), 8: (2 / 5, -1 / 20, 2 / 315, -1 / 2240)}


def _at(f, *shifts):
    """f at the given (offset, axis) pairs."""
    return torch.roll(f, [-n for n, _ in shifts], [a for _, a in shifts])


def _d1(f, a, dx, order):
    return sum(c * (_at(f, (n, a)) - _at(f, (-n, a))) for n, c in enumerate(D1[order], 1)) / dx


def _d2(f, a, b, dx, order):
    if a == b:
        cs = D2[order]
        return (cs[0] * f + sum(c * (_at(f, (n, a)) + _at(f, (-n, a))) for n, c in enumerate(cs[1:], 1))) / dx ** 2
    return sum(c * (_at(f, (n, a), (n, b)) + _at(f, (-n, a), (-n, b)) - _at(f, (n, a), (-n, b)) -
                    _at(f, (-n, a), (n, b))) for n, c in enumerate(DM[order], 1)) / dx ** 2


def _grad(f, dx, order):
    return [_d1(f, a, dx, order) for a in range(3)]


def _hess(f, dx, order):
    return [_d2(f, a, b, dx, order) for a, b in PAIRS]


# ---------------------------------------------------------------------------
# inputs: smooth random fields of a run a little after its start
# ---------------------------------------------------------------------------
def _wavenumbers(shape, device):
    px = torch.fft.fftfreq(shape[0], device=device, dtype=torch.float64) * shape[0]
    py = torch.fft.fftfreq(shape[1], device=device, dtype=torch.float64) * shape[1]
    pz = torch.fft.rfftfreq(shape[2], device=device, dtype=torch.float64) * shape[2]
    return (px[:, None, None] ** 2 + py[None, :, None] ** 2 + pz[None, None, :] ** 2).sqrt()


def _random(shape, gen, rms, power):
    """Gaussian random field, P(k) ~ k^power exp(-(k/kc)^2), kc a quarter of the shortest side's points."""
    k = _wavenumbers(shape, gen.device)
    amp = torch.where(k > 0, k.clamp(min=1.0) ** (power / 2) * torch.exp(-0.5 * (k / (min(shape) / 4.0)) ** 2), 0.0)
    f = torch.fft.irfftn(amp * torch.fft.rfftn(torch.randn(shape, generator=gen, device=gen.device,
                                                           dtype=torch.float64)), s=shape)
    f -= f.mean()
    return f * (rms / f.square().mean().sqrt())


def _inverse_laplacian(f):
    k = _wavenumbers(tuple(f.shape), f.device)
    p2 = (2.0 * math.pi * k) ** 2
    return torch.fft.irfftn(torch.where(p2 > 0, torch.fft.rfftn(f) / -p2.clamp(min=1e-30), 0.0), s=f.shape)


def _box_state(case, shape, seed):
    """The `_p` registers of one box, (fields, nx, ny, nz) on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    matter, order = case["matter"], case["order"]
    dx, _ = _spacing(shape)
    U = torch.zeros((NFIELDS[matter] + (1 if case["z4c"] else 0), *shape), dtype=torch.float64, device="cuda")
    small = 1.0e-6
    if matter == "dust":
        # a Gaussian random density contrast in synchronous gauge: Newtonian potential, curvature, expansion
        # and shear to first order, the density from the Hamiltonian constraint
        delta = _random(shape, gen, 1.0e-4, 0.96)
        pot = _inverse_laplacian(1.5 * delta)
        phi = torch.log1p(-10.0 / 3.0 * pot) / 4.0
        lap = sum(_d2(pot, a, a, dx, order) for a in range(3))
        U[PHI] = phi
        U[K] = -3.0 * (1.0 + 2.0 * pot) + 2.0 / 3.0 * lap
        for q, (i, j) in enumerate(PAIRS):
            U[A + q] = 2.0 / 3.0 * (_d2(pot, i, j, dx, order) - (lap / 3.0 if i == j else 0.0))
        curv = sum(_d2(phi, a, a, dx, order) + _d1(phi, a, dx, order) ** 2 for a in range(3)) * torch.exp(-4.0 * phi)
        rho = (U[K] ** 2 / 12.0 - curv) / (2.0 * math.pi) - LAMBDA
        U[MAT] = torch.exp(6.0 * phi) * rho
        for m in range(3):
            U[MAT + 1 + m] = RHO * _random(shape, gen, small, 0.0)
    elif matter == "scalar":
        # a homogeneous field with fluctuations, the expansion from its energy density
        s = 1.0e-2 + _random(shape, gen, 1.0e-5, -2.0)
        g = _grad(s, dx, order)
        U[MAT] = s
        U[MAT + 1] = _random(shape, gen, 1.0e-4, 0.0)
        for m in range(3):
            U[MAT + 2 + m] = g[m]
        rho = 0.5 * MASS ** 2 * s ** 2 + 0.5 * (g[0] ** 2 + g[1] ** 2 + g[2] ** 2)
        U[K] = -torch.sqrt(24.0 * math.pi * rho)
        U[PHI] = _random(shape, gen, small, -2.0)
    else:
        small = 1.0e-5
        U[PHI] = _random(shape, gen, small, -2.0)
        U[K] = _random(shape, gen, small, 0.0)
    for q in range(6):
        U[G + q] = _random(shape, gen, small, -2.0)
        if matter != "dust":
            U[A + q] = _random(shape, gen, small, 0.0)
    for i in range(3):
        U[GAM + i] = -sum(_d1(U[G + SYM[i][j]], j, dx, order) for j in range(3))
    U[ALPHA] = _random(shape, gen, small, -2.0)
    if case["z4c"]:
        U[-1] = _random(shape, gen, 0.1 * small, 0.0)
    return U


def _box_seed(seed, box):
    return int(seed) * 64 + box


# ---------------------------------------------------------------------------
# a pass through the framework
# ---------------------------------------------------------------------------
class _Memory:
    """__cuda_array_interface__ of memory that a context owns; the tensor made
    from it holds this object, and so the context, for as long as it lives."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 2,
                                         "strides": None}


def _parts(case, U):
    """One box's registers as the groups of fields that belong together."""
    out = {"gamma": U[G:PHI], "phi": U[PHI], "A": U[A:K], "K": U[K], "Gamma": U[GAM:ALPHA], "alpha": U[ALPHA]}
    if case["matter"] == "dust":
        out.update(D=U[MAT], S=U[MAT + 1:MAT + 4])
    elif case["matter"] == "scalar":
        out.update(field=U[MAT], Pi=U[MAT + 1], psi=U[MAT + 2:MAT + 5])
    if case["z4c"]:
        out["theta"] = U[-1]
    return out


def prepare(case, seed):
    states, configs, shapes = [], [], _shapes(case)
    for b, shape in enumerate(shapes):
        dx, dt = _spacing(shape)
        U = _box_state(case, shape, _box_seed(seed, b)).cpu().numpy()
        states.append(BoxState(fields=U, matter=MATTER[case["matter"]], dx=dx, dt=dt, z4c=case["z4c"],
                               lam=LAMBDA if case["matter"] == "dust" else 0.0))
        configs.append(BoxConfig(order=case["order"], lapse=case["lapse"], precision=case["precision"],
                                 potential="quadratic", pot_mass=MASS, ko_coeff=case["ko"]))
    ev = Evolution(states, configs)
    ev.step_init()
    views = []
    for b, shape in enumerate(shapes):
        p = ctypes.POINTER(ctypes.c_double)()
        ev._check(ev.L.cg_device_register(ev.ctx, b, b"p", ctypes.byref(p)))
        ptr = ctypes.cast(p, ctypes.c_void_p).value
        U = torch.as_tensor(_Memory(ev, ptr, (states[b].fields.shape[0], *shape)), device="cuda")
        views.append(_parts(case, U))
    return {"ev": ev, "what": case["what"], "steps": case["steps"], "views": views}


def run(state):
    ev = state["ev"]
    if state["what"] == "constraints":
        return ev.constraints(0)
    ev.step(state["steps"])
    return state["views"]


def work(case):
    """Register traffic of the RK4 substeps (inputs read once and results
    written once each substep) and the arithmetic of the right-hand sides."""
    nf = NFIELDS[case["matter"]] + (1 if case["z4c"] else 0)
    points = sum(x * y * z for x, y, z in _shapes(case))
    r = case["order"] // 2
    # per field with second derivatives: 3 first, 3 second, 3 mixed differences
    stencil = 8 * (3 * (4 * r) + 3 * (4 * r + 1) + 3 * (5 * r)) + 4 * 3 * 4 * r
    matter = {"dust": 4 * 3 * 6 * r + 400, "scalar": 5 * 3 * 4 * r + 150, "vacuum": 0}[case["matter"]]
    flops = stencil + matter + 2600 + 12 * nf
    if case["ko"]:
        flops += 18 * 30
    if case["what"] == "constraints":
        return {"bytes": 8.0 * nf * points, "flops": float(flops * points)}
    if case["precision"] == "mixed":
        # FP32 substep inputs, FP64 registers; (a, p -> f, a), 2 x (a, p, f -> f, a), (a, p, f -> p, a)
        per_step = nf * ((4 + 8 + 8 + 4) + 2 * (4 + 8 + 8 + 8 + 4) + (4 + 8 + 8 + 8 + 4))
    else:
        per_step = 8 * 17 * nf
    return {"bytes": float(case["steps"] * points * per_step), "flops": float(case["steps"] * 4 * flops * points)}


def tolerance(case):
    # four times the distance from exact() over the ranges above: FP32 perturbations 2.6e-7 (K and A of boxes whose
    # means vanish), FP64 1.3e-11 (A and Gamma, second differences of much larger fields)
    return {"rel": 1.0e-6} if case["precision"] == "mixed" and case["what"] == "step" else {"rel": 5.0e-11}


# ---------------------------------------------------------------------------
# the same pass in plain 64-bit torch: BSSN (Z4c) with dust or a scalar field
# ---------------------------------------------------------------------------
def _inverse(g):
    """Inverse of the unit-determinant metric delta + g."""
    return [1 + g[3] + g[5] - g[4] ** 2 + g[3] * g[5], g[2] * g[4] - g[1] * (1 + g[5]), g[1] * g[4] - g[2] * (1 + g[3]),
            1 + g[0] + g[5] - g[2] ** 2 + g[0] * g[5], g[1] * g[2] - g[4] * (1 + g[0]),
            1 + g[0] + g[3] - g[1] ** 2 + g[0] * g[3]]


def _trace(gi, t):
    return gi[0] * t[0] + gi[3] * t[3] + gi[5] * t[5] + 2 * (gi[1] * t[1] + gi[2] * t[2] + gi[4] * t[4])


def _normalised(U):
    """The first substep's input: unit determinant, trace-free A."""
    V = U.clone()
    g = U[G:PHI]
    less1 = (g[0] + g[3] + g[5] - g[1] ** 2 - g[2] ** 2 - g[4] ** 2 + g[0] * g[3] + g[0] * g[5] + g[3] * g[5]
             - g[4] ** 2 * g[0] - g[2] ** 2 * g[3] - g[1] ** 2 * g[5] + 2 * g[1] * g[2] * g[4] + g[0] * g[3] * g[5])
    t = -torch.expm1(torch.log1p(less1) / 3)
    for q, (i, j) in enumerate(PAIRS):
        V[G + q] = (g[q] + (t if i == j else 0.0)) / (1 - t)
    tr = _trace(_inverse(V[G:PHI]), U[A:K])
    for q, (i, j) in enumerate(PAIRS):
        V[A + q] = (U[A + q] - (V[G + q] + (1.0 if i == j else 0.0)) * tr / 3) / (1 - t)
    return V


def _dust(U, gi):
    """Lorentz factor and transport velocity of the dust."""
    S = U[MAT + 1:MAT + 4]
    up = [sum(gi[SYM[i][j]] * S[j] for j in range(3)) for i in range(3)]
    e4 = torch.exp(-4 * U[PHI])
    W = torch.sqrt(1 + e4 * sum(up[i] * S[i] for i in range(3)) / U[MAT] ** 2)
    return W, [torch.exp(-10 * U[PHI]) * up[i] for i in range(3)]


class _Point:
    """Everything the right-hand sides and the constraints share, on one box."""

    def __init__(self, case, U, lag, dx):
        order = case["order"]
        self.U, self.dx, self.order = U, dx, order
        gi = self.gi = _inverse(U[G:PHI])
        gm = self.gm = [U[G + q] + (1.0 if i == j else 0.0) for q, (i, j) in enumerate(PAIRS)]
        self.alpha = 1.0 + U[ALPHA]
        phi, e = U[PHI], torch.exp(-4 * U[PHI])
        self.e = e
        dg = [_grad(U[G + q], dx, order) for q in range(6)]
        self.dg = dg
        GL = self.GL = [[0.5 * (dg[SYM[k][i]][j] + dg[SYM[j][i]][k] - dg[q][i]) for q, (j, k) in enumerate(PAIRS)]
                        for i in range(3)]
        GU = self.GU = [[sum(gi[SYM[i][l]] * GL[l][q] for l in range(3)) for q in range(6)] for i in range(3)]
        Gd = self.Gd = [_trace(gi, GU[i]) for i in range(3)]
        dphi = self.dphi = _grad(phi, dx, order)
        h = _hess(phi, dx, order)
        DDphi = [h[q] - sum(GU[k][q] * dphi[k] for k in range(3)) for q in range(6)]
        lap = _trace(gi, [DDphi[q] + 2 * dphi[i] * dphi[j] for q, (i, j) in enumerate(PAIRS)])
        dGam = [_grad(U[GAM + k], dx, order) for k in range(3)]
        self.R = []
        for q, (i, j) in enumerate(PAIRS):
            r = -0.5 * _trace(gi, _hess(U[G + q], dx, order))
            for k in range(3):
                r = r + 0.5 * (gm[SYM[k][i]] * dGam[k][j] + gm[SYM[k][j]] * dGam[k][i]
                               + Gd[k] * (GL[i][SYM[j][k]] + GL[j][SYM[i][k]]))
                for m in range(3):
                    # the symbols with one index raised by the (l, m) metric
                    Hi = sum(gi[SYM[l][m]] * GU[k][SYM[l][i]] for l in range(3))
                    Hj = sum(gi[SYM[l][m]] * GU[k][SYM[l][j]] for l in range(3))
                    r = r + Hi * GL[j][SYM[k][m]] + Hj * GL[i][SYM[k][m]] \
                        + 0.5 * (Hi * GL[k][SYM[m][j]] + Hj * GL[k][SYM[m][i]])
            self.R.append(r - 2 * (DDphi[q] - 2 * dphi[i] * dphi[j] + gm[q] * lap))
        self.ricci = e * _trace(gi, self.R)
        a = U[A:K]
        self.Au = [sum(gi[SYM[i][x]] * gi[SYM[j][y]] * a[SYM[x][y]] for x in range(3) for y in range(3))
                   for i, j in PAIRS]
        self.AA = self.Au[0] * a[0] + self.Au[3] * a[3] + self.Au[5] * a[5] \
            + 2 * (self.Au[1] * a[1] + self.Au[2] * a[2] + self.Au[4] * a[4])
        self.dK = _grad(U[K], dx, order)
        self.da = _grad(U[ALPHA], dx, order)
        zero = torch.zeros_like(phi)
        self.r, self.s, self.S, self.T = zero, zero, [zero] * 3, [zero] * 6
        if case["matter"] == "dust":
            # the sources pair the Lorentz factor, volume and metric of the
            # previous substep's state with the current density and momentum
            W, _ = _dust(lag, _inverse(lag[G:PHI]))
            vol, e4 = torch.exp(6 * lag[PHI]), torch.exp(4 * lag[PHI])
            D, S = U[MAT], U[MAT + 1:MAT + 4]
            s = D / vol * (W * W - 1) / W
            self.r, self.s = W * D / vol + LAMBDA, s - 3 * LAMBDA
            self.S = [S[i] / vol for i in range(3)]
            self.T = [S[i] * S[j] / (W * D * vol) - e4 * (lag[G + q] + (1.0 if i == j else 0.0)) * s / 3
                      for q, (i, j) in enumerate(PAIRS)]
        elif case["matter"] == "scalar":
            f, Pi = U[MAT], U[MAT + 1]
            d = self.df = _grad(f, dx, order)
            dd = sum(gi[SYM[i][j]] * d[i] * d[j] for i in range(3) for j in range(3))
            V = 0.5 * MASS ** 2 * f ** 2
            self.r, self.s = 0.5 * Pi ** 2 + 0.5 * e * dd + V, 1.5 * Pi ** 2 - 0.5 * e * dd - 3 * V
            self.S = [Pi * d[i] for i in range(3)]
            self.T = [d[i] * d[j] - gm[q] * dd / 3 for q, (i, j) in enumerate(PAIRS)]


def _dissipation(case, f, dx):
    """Kreiss-Oliger term that a right-hand side loses (orders 2 and 8)."""
    if case["order"] == 2:
        cs, scale = (6.0, -4.0, 1.0), case["ko"] / 64 / dx
    else:
        cs, scale = (-252.0, 210.0, -120.0, 45.0, -10.0, 1.0), -case["ko"] / 1024 / dx
    return scale * sum(cs[0] * f + sum(c * (_at(f, (n, a)) + _at(f, (-n, a))) for n, c in enumerate(cs[1:], 1))
                       for a in range(3))


def _rhs(case, U, lag, dx):
    p = _Point(case, U, lag, dx)
    order, gi, gm, al, da, dphi = case["order"], p.gi, p.gm, p.alpha, p.da, p.dphi
    a, k, theta = U[A:K], U[K], U[-1] if case["z4c"] else torch.zeros_like(U[K])
    k1, k2 = (0.5, 0.1) if case["z4c"] else (0.0, 0.0)
    dth = _grad(theta, dx, order) if case["z4c"] else [0.0] * 3
    Kt = k + 2 * theta
    out = torch.empty_like(U)
    h = _hess(U[ALPHA], dx, order)
    gl = [sum(gi[SYM[i][j]] * dphi[j] for j in range(3)) for i in range(3)]
    DDa = []
    for q, (i, j) in enumerate(PAIRS):
        t = h[q] - 2 * (da[i] * dphi[j] + da[j] * dphi[i])
        for l in range(3):
            t = t - (p.GU[l][q] - 2 * gm[q] * gl[l]) * da[l]
        DDa.append(t)
    tr = _trace(gi, DDa)
    for q, (i, j) in enumerate(PAIRS):
        aa = sum(gi[SYM[x][y]] * a[SYM[x][i]] * a[SYM[y][j]] for x in range(3) for y in range(3))
        out[G + q] = -2 * al * a[q]
        out[A + q] = p.e * (al * (p.R[q] - 8 * math.pi * p.T[q]) - DDa[q] + gm[q] * tr / 3) \
            - al * gm[q] * p.ricci / 3 + al * (Kt * a[q] - 2 * aa)
    for i in range(3):
        au = [p.Au[SYM[i][j]] for j in range(3)]
        t = sum((2 if x != y else 1) * p.GU[i][q] * p.Au[q] for q, (x, y) in enumerate(PAIRS))
        for j in range(3):
            t = t + 6 * au[j] * dphi[j] - gi[SYM[i][j]] * ((2 * p.dK[j] + dth[j]) / 3 + 8 * math.pi * p.S[j])
        out[GAM + i] = 2 * al * (t - 2 * al * k1 * (U[GAM + i] - p.Gd[i])) - 2 * sum(au[j] * da[j] for j in range(3))
    out[K] = -p.e * tr + al * (Kt * Kt / 3 + p.AA) + 4 * math.pi * al * (p.r + p.s) + k1 * (1 - k2) * theta
    out[PHI] = -al * Kt / 6
    if case["lapse"] == "OnePlusLog":
        w = torch.exp(6 * U[PHI])
        out[ALPHA] = -2 * al * (k - (w * k).sum() / w.sum())
    else:
        out[ALPHA] = -al * k
    if case["z4c"]:
        out[-1] = 0.5 * al * (p.ricci + 2 / 3 * Kt * Kt - p.AA - 16 * math.pi * p.r) - al * k1 * (2 + k2) * theta
    if case["matter"] == "dust":
        W, v = _dust(U, gi)
        D = U[MAT]
        out[MAT] = sum(_d1(al * D * v[i], i, dx, order) for i in range(3))
        for m in range(3):
            s = sum(v[i] * v[j] * (4 * gm[SYM[i][j]] * dphi[m] + p.dg[SYM[i][j]][m])
                    for i in range(3) for j in range(3))
            out[MAT + 1 + m] = sum(_d1(al * U[MAT + 1 + m] * v[i], i, dx, order) for i in range(3)) \
                + 0.5 * al * W * D * torch.exp(4 * U[PHI]) * s - W * D * da[m]
    elif case["matter"] == "scalar":
        Pi, psi = U[MAT + 1], U[MAT + 2:MAT + 5]
        out[MAT] = -al * Pi
        t = al * (k * Pi + MASS ** 2 * U[MAT])
        dpsi = [_grad(psi[m], dx, order) for m in range(3)]
        dPi = _grad(Pi, dx, order)
        for i in range(3):
            t = t + al * p.e * (U[GAM + i] - 2 * gl[i]) * psi[i]
            for j in range(3):
                t = t - p.e * gi[SYM[i][j]] * (al * dpsi[j][i] + psi[i] * da[j])
            out[MAT + 2 + i] = -al * dPi[i] - Pi * da[i]
        out[MAT + 1] = t
    if case["ko"]:
        for f in list(range(MAT)) + ([U.shape[0] - 1] if case["z4c"] else []):
            out[f] -= _dissipation(case, U[f], dx)
    return out


def _constraints(case, U, dx):
    """H, M, G, A, S: mean, standard deviation, largest, sum of the scales,
    the same of the scaled values; H and M their L2 norms too."""
    p = _Point(case, U, U, dx)
    gi, a, g, e6 = p.gi, U[A:K], U[G:PHI], torch.exp(6 * U[PHI])
    k2, rho = 2 / 3 * U[K] ** 2, 16 * math.pi * p.r
    e5 = torch.exp(5 * U[PHI]) / 8
    H = -e5 * (p.ricci + k2 - p.AA - rho), e5 * (p.ricci ** 2 + p.AA ** 2 + k2 ** 2 + rho ** 2).sqrt()
    dA = [_grad(a[q], dx, case["order"]) for q in range(6)]
    m2, ms2, c2, cs2 = 0.0, 0.0, 0.0, 0.0
    for i in range(3):
        t6 = sum(gi[SYM[x][d]] * a[SYM[x][i]] * p.dphi[d] for x in range(3) for d in range(3))
        t = sum(gi[SYM[x][d]] * dA[SYM[x][i]][d] for x in range(3) for d in range(3))
        for x in range(3):
            t = t - p.Gd[x] * a[SYM[x][i]]
            for y in range(3):
                t = t - p.GL[y][SYM[x][i]] * p.Au[SYM[x][y]]
        k, s = 2 / 3 * p.dK[i], 8 * math.pi * p.S[i]
        m2 = m2 + (e6 * (6 * t6 + t - k - s)) ** 2
        ms2 = ms2 + (e6 * (k.abs() + s.abs() + 6 * t6.abs() + t.abs())) ** 2
        Gu = p.GU[i]
        c2 = c2 + (U[GAM + i] - p.Gd[i]) ** 2
        rest = gi[0] * Gu[0] - gi[3] * Gu[3] - gi[5] * Gu[5] - 2 * (gi[1] * Gu[1] + gi[2] * Gu[2] + gi[4] * Gu[4])
        cs2 = cs2 + (U[GAM + i].abs() + rest.abs()) ** 2
    tr = [gi[q] * a[q] for q in range(6)]
    det = (g[0] + g[3] + g[5], g[1] ** 2 + g[2] ** 2 + g[4] ** 2, g[0] * g[3], g[0] * g[5], g[3] * g[5],
           g[4] ** 2 * g[0] + g[2] ** 2 * g[3] + g[1] ** 2 * g[5], 2 * g[1] * g[2] * g[4], g[0] * g[3] * g[5])
    less1 = det[0] - det[1] + det[2] + det[3] + det[4] - det[5] + det[6] + det[7]
    scale = g[0].abs() + g[3].abs() + g[5].abs() + det[1] + det[2].abs() + det[3].abs() + det[4].abs() + det[5] \
        + det[6].abs() + det[7].abs()
    values = {"H": H, "M": (m2.sqrt(), ms2.sqrt()), "G": (c2.sqrt(), cs2.sqrt()),
              "A": (_trace(gi, a), tr[0].abs() + tr[3].abs() + tr[5].abs()
                    + 2 * (tr[1].abs() + tr[2].abs() + tr[4].abs())),
              "S": (less1.abs(), scale)}
    out = {}
    for name, (v, s) in values.items():
        r = v / s
        o = [v.mean(), v.std(), v.abs().max(), s.sum(), r.mean(), r.std(), r.abs().max()]
        if name in "HM":
            o.append((v.square().sum() * dx ** 3).sqrt())
        out[name] = np.array([float(x) for x in o])
    # A and S vanish but for rounding: their values have no 64-bit reference
    return {k: v if k in "HMG" else None for k, v in out.items()}


def exact(case, seed):
    out = []
    for b, shape in enumerate(_shapes(case)):
        dx, dt = _spacing(shape)
        p = _box_state(case, shape, _box_seed(seed, b))
        if case["what"] == "constraints":
            return _constraints(case, _normalised(p), dx)
        for _ in range(case["steps"]):
            a = _normalised(p)
            lag, new = a, p.clone()
            for weight, ahead in ((1 / 6, 1 / 2), (1 / 3, 1 / 2), (1 / 3, 1.0), (1 / 6, 0.0)):
                k = _rhs(case, a, lag, dx)
                new.add_(k, alpha=weight * dt)
                lag, a = a, p.add(k, alpha=ahead * dt)
            p = new
        out.append(_parts(case, p))
    return out
