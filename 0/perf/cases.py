"""Performance cases: the calls a user of the time step makes, with their inputs.

Three kinds of pass:

``solve``   upload a state, run the device-resident driver loop for a number
            of steps, download the result: one leg of a production run.
``dropin``  dt = cfl x getCourantTimestep, then SolutionScheme::advance on the
            caller's host array, a number of times: what a driver of the
            reference does when it swaps the scheme.
``batch``   a server's queue of independent grids: admit all, step until all
            have reached their end time, retire all.

``exact`` integrates the same scheme in 64-bit torch, written from the
published methods (Godunov / MUSCL with the generalised minmod, WENO5 with
Shen and Zha's indicators, HLLE, HLLC, Toth's flux CT, Antón's (Z, W) Newton
iteration), without this package's code.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mara2_gb300.batch import Batch
from mara2_gb300.scheme import Scheme
from mara2_gb300.solver import Solver

NQ = {"hydro": 5, "mhd": 8, "rmhd": 8}
GUARD = {"pcm": 1, "plm": 2, "weno5": 3}
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def _case(kind, problem, shape, recon, riemann, bc, rk, precision, steps, **more):
    law = {"tube": "hydro", "shear": "hydro", "turbulence": "mhd", "blast": "rmhd"}[problem]
    nx, ny, nz = shape
    return dict(kind=kind, problem=problem, law=law, nx=nx, ny=ny, nz=nz, recon=recon, riemann=riemann, bc=bc, rk=rk,
                precision=precision, steps=steps, **more)


def listed():
    return [
        # the regression shock tube: the smallest grid, a chain of launches
        dict(_case("solve", "tube", (1024, 1, 1), "plm", "hlle", "outflow", 2, "fp64", 64), name="tube-1024-fp64"),
        # a long, odd-sized tube in the fast precision
        dict(_case("solve", "tube", (4099, 1, 1), "plm", "hllc", "outflow", 2, "mixed", 256), name="tube-4099-mixed"),
        # Kelvin-Helmholtz at its benchmark size: the default precision ...
        dict(_case("solve", "shear", (1024, 1024, 1), "plm", "hllc", "periodic", 2, "fp64", 4), name="shear-1024-fp64"),
        # ... and the fast one
        dict(_case("solve", "shear", (1024, 1024, 1), "plm", "hllc", "periodic", 2, "mixed", 32),
             name="shear-1024-mixed"),
        # a ragged 2-D grid with open boundaries and the FP64 accumulator
        dict(_case("solve", "shear", (1531, 877, 1), "plm", "hllc", "outflow", 3, "mixed_fp64", 16),
             name="shear-1531x877-acc64"),
        # 3-D hydrodynamics in a closed box, ragged
        dict(_case("solve", "shear", (112, 90, 75), "plm", "hlle", "reflecting", 3, "mixed", 16),
             name="shear3d-112x90x75-mixed"),
        # MHD turbulence with constrained transport
        dict(_case("solve", "turbulence", (128, 128, 128), "plm", "hlle", "periodic", 3, "mixed", 8),
             name="turbulence-128-mixed"),
        # a reference MHD driver with the scheme swapped: default precision, its own pageable array
        dict(_case("dropin", "turbulence", (64, 56, 48), "plm", "hlle", "periodic", 3, "fp64", 2, pinned=False),
             name="turbulence-64x56x48-dropin"),
        # relativistic MHD blast wave, WENO5
        dict(_case("solve", "blast", (512, 512, 1), "weno5", "hlle", "outflow", 3, "mixed", 16), name="blast-512-mixed"),
        # the same physics in the default precision, a small ragged grid
        dict(_case("solve", "blast", (160, 131, 1), "weno5", "hlle", "outflow", 3, "fp64", 2), name="blast-160x131-fp64"),
        # the drop-in call on a large page-locked array
        dict(_case("dropin", "shear", (2048, 2048, 1), "plm", "hllc", "periodic", 2, "mixed", 1, pinned=True),
             name="shear-2048-dropin-mixed"),
        # a server's queue of uneven 1-D and 2-D shock problems
        dict(_case("batch", "tube", (2048, 384, 1), "plm", "hllc", "outflow", 2, "mixed", 0, grids=24, t_final=0.01),
             name="batch-24-mixed"),
    ]


# zones x RK stages x axes per second to size the drawn cases by (orders of magnitude; WENO5 takes longer)
_RATE = {("hydro", "fp64"): 1e9, ("mhd", "fp64"): 5e8, ("rmhd", "fp64"): 4e7,
         ("hydro", "mixed"): 2.5e10, ("mhd", "mixed"): 1.5e10, ("rmhd", "mixed"): 4e9,
         ("hydro", "mixed_fp64"): 2e10, ("mhd", "mixed_fp64"): 1.5e10, ("rmhd", "mixed_fp64"): 1e9}
_WENO = {"fp64": 0.35, "mixed": 0.6, "mixed_fp64": 0.6}
# a stage along one axis takes at least this long, however small the grid
_LATENCY = {("hydro", "fp64"): 5e-5, ("mhd", "fp64"): 1e-4, ("rmhd", "fp64"): 6e-4, ("hydro", "mixed"): 5e-6,
            ("mhd", "mixed"): 1e-5, ("rmhd", "mixed"): 2e-5, ("hydro", "mixed_fp64"): 8e-6, ("mhd", "mixed_fp64"): 1e-5,
            ("rmhd", "mixed_fp64"): 1e-4}
_PASS = 8e-3  # seconds


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    problem = rng.choice(["tube", "shear", "shear", "turbulence", "blast", "batch"])
    precision = rng.choice(["fp64", "mixed", "mixed", "mixed_fp64"])
    if problem == "batch":
        return _case("batch", "tube", (_log(rng, 512, 2048), _log(rng, 160, 384), 1), "plm", rng.choice(["hlle", "hllc"]),
                     "outflow", 2, "mixed", 0, grids=rng.randint(6, 24), t_final=round(rng.uniform(0.002, 0.01), 5))
    law = {"tube": "hydro", "shear": "hydro", "turbulence": "mhd", "blast": "rmhd"}[problem]
    recon = rng.choice(["plm", "plm", "weno5", "pcm"])
    riemann = rng.choice(["hlle", "hllc"]) if law == "hydro" else "hlle"
    rk = rng.choice([1, 2, 3]) if recon == "pcm" else rng.choice([2, 3])
    if problem == "tube":
        shape, bc = (_log(rng, 128, 16384), 1, 1), rng.choice(["outflow", "reflecting"])
    elif problem == "blast":
        shape, bc = (_log(rng, 48, 512), _log(rng, 48, 512), 1), rng.choice(["outflow", "periodic"])
    elif problem == "turbulence":
        shape, bc = (_log(rng, 24, 128), _log(rng, 24, 128), _log(rng, 24, 128)), "periodic"
        if rng.random() < 0.3:
            shape = (_log(rng, 64, 1024), _log(rng, 64, 1024), 1)
    else:
        shape, bc = (_log(rng, 64, 1536), _log(rng, 64, 1536), 1), rng.choice(["periodic", "outflow", "reflecting"])
        if rng.random() < 0.35:
            shape = (_log(rng, 24, 128), _log(rng, 24, 128), _log(rng, 24, 128))
    slower = 1 / _WENO[precision] if recon == "weno5" and law != "rmhd" else 1.0
    rate, least = _RATE[law, precision] / slower, _LATENCY[law, precision] * slower
    dims = sum(n > 1 for n in shape)

    def seconds(n):
        return rk * dims * max(n[0] * n[1] * n[2] / rate, least)
    # a pass of at most about _PASS seconds
    while seconds(shape) > _PASS:
        shape = tuple(n if n == 1 else int(n * 0.9) for n in shape)
    steps = max(1, min(128, int(_PASS / seconds(shape))))
    if problem != "tube" and rng.random() < 0.25:
        return _case("dropin", problem, shape, recon, riemann, bc, rk, precision, min(steps, 2),
                     pinned=rng.random() < 0.5)
    return _case("solve", problem, shape, recon, riemann, bc, rk, precision, steps)


# ---- inputs -------------------------------------------------------------------
def _scheme(case, shape=None):
    shape = shape or (case["nx"], case["ny"], case["nz"])
    box = {"blast": 6.0}.get(case["problem"])
    return Scheme(law=case["law"], recon=case["recon"], riemann=case["riemann"], bc=case["bc"], rk_order=case["rk"],
                  shape=shape, lower=(-box, -box, 0.0) if box else (0.0, 0.0, 0.0),
                  upper=(box, box, 1.0) if box else (1.0, 1.0, 1.0),
                  gamma=4.0 / 3 if case["law"] == "rmhd" else 5.0 / 3, plm_theta=1.5,
                  cfl=0.3 if case["law"] != "hydro" else 0.4)


def _centres(s):
    x = [torch.linspace(0.5, n - 0.5, n, dtype=torch.float64, device=DEVICE) * ((u - lo) / n) + lo
         for n, lo, u in zip(s.shape, s.lower, s.upper)]
    return torch.meshgrid(*x, indexing="ij")


def _waves(s, r, rms, count=12, kmax=3):
    """A smooth random periodic 3-vector field of the given rms magnitude."""
    x = [(c - lo) / (u - lo) for c, lo, u in zip(_centres(s), s.lower, s.upper)]
    v = torch.zeros((3,) + s.shape, dtype=torch.float64, device=DEVICE)
    for _ in range(count):
        k = [int(r.integers(-kmax, kmax + 1)) if n > 1 else 0 for n in s.shape]
        wave = torch.cos(2 * math.pi * (k[0] * x[0] + k[1] * x[1] + k[2] * x[2] + r.random()))
        for c in range(3):
            v[c] += (r.random() - 0.5) * wave
    return v * (rms / max(float(v.square().sum(0).mean().sqrt()), 1e-30))


def _curl(s, A):
    """curl A by centred differences on a periodic grid: its centred divergence is zero to rounding."""
    def d(f, a):
        n = s.shape[a]
        if n == 1:
            return torch.zeros_like(f)
        return (torch.roll(f, -1, a) - torch.roll(f, 1, a)) * (n / (2 * (s.upper[a] - s.lower[a])))
    return torch.stack([d(A[2], 1) - d(A[1], 2), d(A[0], 2) - d(A[2], 0), d(A[1], 0) - d(A[0], 1)])


def _interior(case, s, seed):
    """The initial primitives of the interior zones, (nq, ni, nj, nk)."""
    r = np.random.default_rng(seed)
    x, y, z = _centres(s)
    P = torch.zeros((NQ[case["law"]],) + s.shape, dtype=torch.float64, device=DEVICE)
    if case["problem"] == "tube":
        # two constant states; on 2-D grids the interface passes the centre at a random angle
        a = 2 * math.pi * r.random() if s.shape[1] > 1 else 0.0
        left = ((x - 0.5) * math.cos(a) + (y - 0.5) * math.sin(a)) < 0
        for q, (lo, hi) in enumerate([(0.1, 10), (-0.3, 0.3), (-0.3, 0.3), (0, 0), (0.1, 10)]):
            u = r.random(2)
            v = lo * (hi / lo) ** u if q in (0, 4) else lo + (hi - lo) * u
            P[q] = torch.where(left, float(v[0]), float(v[1]))
    elif case["problem"] == "shear":
        # a shear layer with a seeded perturbation of the velocity
        band = (y - 0.5).abs() < 0.25
        P[0] = torch.where(band, 2.0, 1.0)
        P[1] = torch.where(band, 0.5, -0.5)
        noise = torch.from_numpy(r.uniform(-0.01, 0.01, s.shape)).to(DEVICE)
        P[2] = noise
        if s.shape[2] > 1:
            P[3] = noise.flip(0)
        P[4] = 2.5
    elif case["problem"] == "turbulence":
        # smooth random flow and a divergence-free random field
        P[0], P[4] = 1.0, 1.0
        P[1:4] = _waves(s, r, 0.1)
        B = _curl(s, _waves(s, r, 1.0))
        P[5:8] = B * (0.5 / float(B.square().sum(0).mean().sqrt()))
    else:
        # a hot cylinder in a weakly turbulent, magnetised medium
        P[0] = 0.01
        P[1:4] = _waves(s, r, 0.1)
        P[4] = torch.where((x * x + y * y).sqrt() < 0.8 + 0.8 * r.random(), 1.0, 0.01)
        a = 2 * math.pi * r.random()
        P[5], P[6] = 0.1 * math.cos(a), 0.1 * math.sin(a)
    return P


def _pad(P, bc, g):
    """Guard zones of width g on every axis with more than one zone, axis by axis."""
    for a in range(3):
        n = P.shape[1 + a]
        if n == 1:
            continue
        P = P.movedim(1 + a, 1)
        if bc == "periodic":
            lo, hi = P[:, n - g:], P[:, :g]
        elif bc == "outflow":
            lo, hi = P[:, :1].expand(-1, g, -1, -1), P[:, -1:].expand(-1, g, -1, -1)
        else:
            lo, hi = P[:, :g].flip(1).clone(), P[:, n - g:].flip(1).clone()
            lo[1 + a] *= -1
            hi[1 + a] *= -1
        P = torch.cat([lo, P, hi], 1).movedim(1, 1 + a)
    return P


def _host_state(case, s, seed, pinned):
    P = _pad(_interior(case, s, seed), s.bc, s.stencil).permute(1, 2, 3, 0).contiguous().cpu()
    return (P.pin_memory() if pinned else P).numpy()


def _grids(case):
    """The schemes of a server's queue: half 1-D, half 2-D, sizes log-uniform (the same for every seed)."""
    r = np.random.default_rng(case["nx"] * 4096 + case["ny"])
    out = []
    for k in range(case["grids"]):
        lo, hi = (256, case["nx"]) if k % 2 == 0 else (128, case["ny"])
        n = int(round(lo * (hi / lo) ** r.random()))
        out.append(_scheme(case, (n, 1, 1) if k % 2 == 0 else (n, n, 1)))
    return out


def prepare(case, seed):
    if case["kind"] == "batch":
        grids = [(s, _host_state(case, s, 1000 * seed + k, False)) for k, s in enumerate(_grids(case))]
        zones = sum(s.zones for s, _ in grids)
        cells = max(P.size // 5 for _, P in grids)
        b = Batch(budget_bytes=200 * zones + (1 << 26), max_grids=case["grids"] + 8, max_zones_per_grid=cells,
                  riemann=case["riemann"])
        return {"case": case, "batch": b, "grids": grids}
    s = _scheme(case)
    pinned = case.get("pinned", True)
    P = _host_state(case, s, seed, pinned)
    solver = Solver(s, case["precision"])
    out = None
    if case["kind"] == "solve":
        out = torch.empty(P.shape, dtype=torch.float64).pin_memory().numpy()
    else:
        solver.upload(P)
    return {"case": case, "solver": solver, "P": P, "out": out}


# ---- the pass -----------------------------------------------------------------
def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        slots = {b.admit(s, P, case["t_final"]): k for k, (s, P) in enumerate(state["grids"])}
        done = {}
        while len(done) < len(slots):
            b.step(32)
            for slot in b.poll():
                k = slots[slot]
                done[k] = b.retire(slot, state["grids"][k][0].full_shape)
        return {"P": [done[k][0] for k in range(len(done))],
                "t": np.array([done[k][1] for k in range(len(done))]),
                "steps": np.array([done[k][2] for k in range(len(done))])}
    solver = state["solver"]
    if case["kind"] == "dropin":
        for _ in range(case["steps"]):
            dt = solver.scheme.cfl * solver.courant()
            solver.advance_host(state["P"], dt)
        return {"P": state["P"], "dt": dt}
    solver.upload(state["P"])
    solver.t = 0.0
    solver.run(case["steps"])
    return {"P": solver.download(state["out"]), "t": solver.t}


# operations of one zone-update per RK stage and axis, and per RK stage besides:
# a face's reconstruction, two states and the Riemann solver; the update
_FLOPS = {"hydro": (150, 60), "mhd": (330, 110), "rmhd": (900, 400)}


def work(case):
    """Bytes: the state in and out once per call (8 bytes a value in every precision).  Operations: counted from the
    formulas, each shared value once."""
    if case["kind"] == "batch":
        # the steps a grid takes depend on its states; a typical signal speed of 3
        byts = flops = 0.0
        for s in _grids(case):
            steps = case["t_final"] * 3.0 * s.shape[0] / s.cfl
            byts += s.zones * 5 * 8 * 2
            flops += steps * s.zones * case["rk"] * (s.dims * _FLOPS["hydro"][0] + _FLOPS["hydro"][1])
        return {"bytes": byts, "flops": flops}
    s = _scheme(case)
    face, zone = _FLOPS[case["law"]]
    calls = case["steps"] if case["kind"] == "dropin" else 1
    return {"bytes": 2 * s.zones * NQ[case["law"]] * 8 * calls,
            "flops": case["steps"] * case["rk"] * s.zones * (s.dims * face + zone)}


# ---- the same in 64-bit torch ---------------------------------------------------
def _dot(u, v):
    return u[0] * v[0] + u[1] * v[1] + u[2] * v[2]


def _minmod(theta, l, c, r):
    a, b, d = theta * (c - l), 0.5 * (r - l), theta * (r - c)
    m = torch.minimum(torch.minimum(a.abs(), b.abs()), d.abs())
    return 0.25 * (a.sign() + b.sign()).abs() * (a.sign() + d.sign()) * m


def _weno5(v, A):
    """The value at the right edge of the centre of five points (Jiang and Shu 1996; indicators after Shen and Zha 2010)."""
    p = [(2 * v[2] + 5 * v[3] - v[4]) / 6, (-v[1] + 5 * v[2] + 2 * v[3]) / 6, (2 * v[0] - 7 * v[1] + 11 * v[2]) / 6]
    b = [13 / 12 * (v[2] - 2 * v[3] + v[4]) ** 2 + (3 * v[2] - 4 * v[3] + v[4]) ** 2 / 4,
         13 / 12 * (v[1] - 2 * v[2] + v[3]) ** 2 + (v[1] - v[3]) ** 2 / 4,
         13 / 12 * (v[0] - 2 * v[1] + v[2]) ** 2 + (v[0] - 4 * v[1] + 3 * v[2]) ** 2 / 4]
    lo = torch.minimum(torch.minimum(b[0], b[1]), b[2])
    hi = torch.maximum(torch.maximum(b[0], b[1]), b[2])
    add = lo / (hi + 1e-10) * A * lo
    w = [d / (1e-10 + x + add) ** 2 for d, x in zip((0.3, 0.6, 0.1), b)]
    return (w[0] * p[0] + w[1] * p[1] + w[2] * p[2]) / (w[0] + w[1] + w[2])


def _edges(P, recon):
    """The states on both sides of the faces along axis 1 (last spatial axes kept); n + 1 faces for n interior zones."""
    g = GUARD[recon]
    m = P.shape[1] - 2 * g + 1
    v = [P[:, c:c + m] for c in range(2 * g)]
    if recon == "pcm":
        return v[0], v[1]
    if recon == "plm":
        return v[1] + 0.5 * _minmod(1.5, v[0], v[1], v[2]), v[2] - 0.5 * _minmod(1.5, v[1], v[2], v[3])
    return _weno5(v[:5], 50.0), _weno5(v[:0:-1], 50.0)


def _quartic_range(c4, c3, c2, c1, c0):
    """The smallest and the largest real root (Ferrari's method over the resolvent cubic)."""
    a, b, c, d = c3 / c4, c2 / c4, c1 / c4, c0 / c4
    p2, p1, p0 = -b, c * a - 4 * d, 4 * d * b - c * c - d * a * a
    q, r = p1 / 3 - p2 * p2 / 9, (p1 * p2 - 3 * p0) / 6 - p2 ** 3 / 27
    disc = q ** 3 + r * r

    def cbrt(t):
        return t.sign() * t.abs() ** (1 / 3)
    sd = disc.clamp(min=0).sqrt()
    one = cbrt(r + sd) + cbrt(r - sd)
    three = 2 * (-q).clamp(min=0).sqrt() * torch.cos(
        torch.acos((r / (-q).clamp(min=1e-300).pow(1.5)).clamp(-1, 1)) / 3)
    u = torch.where(disc > 0, one, three) - p2 / 3
    R2 = a * a / 4 + u - b
    R = R2.clamp(min=0).sqrt()
    k = 0.75 * a * a - 2 * b
    m = torch.where(R > 0, (4 * a * b - 8 * c - a ** 3) / (4 * R.clamp(min=1e-300)),
                    2 * (u * u - 4 * d).clamp(min=0).sqrt())
    D2, E2 = k - R2 + m, k - R2 - m
    inf = torch.full_like(a, math.inf)
    D, E = D2.clamp(min=0).sqrt(), E2.clamp(min=0).sqrt()
    lo = torch.minimum(torch.where(D2 >= 0, -a / 4 + R / 2 - D / 2, inf), torch.where(E2 >= 0, -a / 4 - R / 2 - E / 2, inf))
    hi = torch.maximum(torch.where(D2 >= 0, -a / 4 + R / 2 + D / 2, -inf), torch.where(E2 >= 0, -a / 4 - R / 2 + E / 2, -inf))
    return lo, hi


def _state(law, gamma, P, a, need="UFA"):
    """Conserved densities, fluxes along axis a and the extreme wave speeds."""
    rho, v, p = P[0], P[1:4], P[4]
    vn, vv = v[a], _dot(v, v)
    if law == "hydro":
        U = torch.stack([rho, rho * v[0], rho * v[1], rho * v[2], 0.5 * rho * vv + p / (gamma - 1)])
        if need == "U":
            return U
        F = vn * U
        F[1 + a] += p
        F[4] += vn * p
        cs = (gamma * p / rho).sqrt()
        return U, F, vn - cs, vn + cs
    B = P[5:8]
    BB, Bv, Bn = _dot(B, B), _dot(B, v), B[a]
    if law == "mhd":
        U = torch.cat([rho[None], rho * v, (0.5 * rho * vv + 0.5 * BB + p / (gamma - 1))[None], B])
        if need == "U":
            return U
        ps = p + 0.5 * BB
        F = torch.cat([vn * U[:1], vn * U[1:4] - Bn * B, (vn * (U[4] + ps) - Bn * Bv)[None], vn * B - Bn * v])
        F[1 + a] += ps
        c2, a2, n2 = gamma * p / rho, BB / rho, Bn * Bn / rho
        cf = (0.5 * (c2 + a2 + ((c2 + a2) ** 2 - 4 * c2 * n2).clamp(min=0).sqrt())).sqrt()
        return U, F, vn - cf, vn + cf
    W2 = 1 / (1 - vv)
    W = W2.sqrt()
    b0 = W * Bv
    bb = (BB + b0 * b0) / W2
    b = B / W + b0 * v
    bn = b[a]
    ps = p + 0.5 * bb
    h = 1 + p / rho * (gamma / (gamma - 1))
    w = (rho * h + bb) * W2
    D = rho * W
    U = torch.cat([D[None], w * v - b0 * b, (w - ps - b0 * b0 - D)[None], B])
    if need == "U":
        return U
    F = torch.cat([vn * U[:1], vn * U[1:4] - Bn / W * b, (vn * U[4] - Bn * b0 / W + ps * vn)[None], vn * B - Bn * v])
    F[1 + a] += ps
    # fast magnetosonic speeds: the quartic of Anile; Alfven speeds beside them
    c2 = gamma * p / (rho * h)
    K, L = W2 * W2 * rho * h * (1 / c2 - 1), -W2 * (rho * h + bb / c2)
    lo, hi = _quartic_range(K - L - b0 * b0, -4 * K * vn + 2 * L * vn + 2 * b0 * bn,
                            6 * K * vn ** 2 + L * (1 - vn ** 2) + b0 * b0 - bn * bn,
                            -4 * K * vn ** 3 - 2 * L * vn - 2 * b0 * bn, K * vn ** 4 + L * vn ** 2 + bn * bn)
    C = (h + bb).sqrt()
    m, q = (bn - C * vn * W) / (b0 - C * W), (bn + C * vn * W) / (b0 + C * W)
    return (U, F, torch.minimum(torch.minimum(lo, vn), torch.minimum(m, q)),
            torch.maximum(torch.maximum(hi, vn), torch.maximum(m, q)))


def _riemann(law, solver, gamma, PL, PR, a):
    UL, FL, lL, hL = _state(law, gamma, PL, a)
    UR, FR, lR, hR = _state(law, gamma, PR, a)
    ap, am = torch.maximum(hL, hR).clamp(min=0), torch.minimum(lL, lR).clamp(max=0)
    if solver == "hlle":
        return (ap * FL - am * FR + ap * am * (UR - UL)) / (ap - am)
    vl, vr = PL[1 + a], PR[1 + a]
    ml, mr = PL[0] * (am - vl), PR[0] * (ap - vr)
    c = ((PR[4] - mr * vr) - (PL[4] - ml * vl)) / (ml - mr)

    def star(P, U, F, s, vn, m):
        us = U.clone()
        f = m / (s - c)
        us[0] = f
        us[1:4] = f * P[1:4]
        us[1 + a] = f * c
        us[4] = f * (U[4] / P[0] + (c - vn) * (c + P[4] / m))
        return F + s * (us - U)
    F = torch.where(c >= 0, star(PL, UL, FL, am, vl, ml), star(PR, UR, FR, ap, vr, mr))
    F = torch.where(am >= 0, FL, F)
    return torch.where(ap < 0, FR, F)


def _recover(law, gamma, U, P):
    """Primitives of conserved densities; P: the previous ones, a starting point for the relativistic root."""
    Q = torch.empty_like(U)
    if law != "rmhd":
        Q[0] = U[0]
        Q[1:4] = U[1:4] / U[0]
        e = U[4] - 0.5 * _dot(U[1:4], U[1:4]) / U[0]
        if law == "mhd":
            Q[5:8] = U[5:8]
            e = e - 0.5 * _dot(U[5:8], U[5:8])
        Q[4] = e * (gamma - 1)
        return Q
    D, S, T, B = U[0], U[1:4], U[4], U[5:8]
    S2, B2, BS = _dot(S, S), _dot(B, B), _dot(B, S)
    g = (gamma - 1) / gamma
    Z = (S2 + D * D).sqrt()
    W = Z / D
    for _ in range(60):
        f0 = -S2 + (Z + B2) ** 2 * (1 - 1 / W ** 2) - (2 * Z + B2) * BS ** 2 / Z ** 2
        f1 = -T + Z + B2 - (Z / W ** 2 - D / W) * g - 0.5 * B2 / W ** 2 - 0.5 * BS ** 2 / Z ** 2 - D
        a00 = 2 * (B2 + Z) * (BS ** 2 / Z ** 3 + 1 - 1 / W ** 2)
        a01 = 2 * (B2 + Z) ** 2 / W ** 3
        a10 = 1 + BS ** 2 / Z ** 3 - g / W ** 2
        a11 = B2 / W ** 3 + (2 * Z - D * W) / W ** 3 * g
        det = a00 * a11 - a01 * a10
        dZ, dW = -(a11 * f0 - a01 * f1) / det, -(a00 * f1 - a10 * f0) / det
        Z, W = (Z + dZ).abs(), (W + dW).clamp(1.0, 1e12)
        if float((dZ / Z).abs().add((dW / W).abs()).max()) < 1e-14:
            break
    Q[0] = D / W
    Q[4] = (Z / W ** 2 - D / W) * g
    Q[1:4] = (S + BS / Z * B) / (Z + B2)
    Q[5:8] = B
    return Q


def _courant(case, s, P):
    fastest = 0.0
    for a in range(3):
        _, _, lo, hi = _state(case["law"], s.gamma, P, a)
        fastest = max(fastest, float(lo.abs().max()), float(hi.abs().max()))
    return min((u - lo) / n for u, lo, n in zip(s.upper, s.lower, s.shape)) / fastest


def _ct(F, axes):
    """Toth's flux CT (2000, eq. 25): a corrected flux is the mean of the EMFs on its face's two edges.  F[a] covers
    the faces of axis a over the zones with one guard on the other axes."""
    def cut(f, a, lo, hi):
        return f.narrow(a, lo, f.shape[a] - lo - hi)
    G = {a: F[a].clone() for a in axes}
    for a in axes:
        G[a][5 + a] = 0
    for a in axes:
        for b in axes:
            if b <= a:
                continue
            # a guard-extended axis t has zones -1 .. n; faces 0 .. n of axis t lie between zones t-1 and t
            fa, fb = F[a][5 + b], F[b][5 + a]
            E = 0.25 * (cut(fa, b, 1, 0) + cut(fa, b, 0, 1) - cut(fb, a, 1, 0) - cut(fb, a, 0, 1))
            G[a][5 + b].narrow(b, 1, fa.shape[b] - 2).copy_(0.5 * (cut(E, b, 1, 0) + cut(E, b, 0, 1)))
            G[b][5 + a].narrow(a, 1, fb.shape[a] - 2).copy_(-0.5 * (cut(E, a, 1, 0) + cut(E, a, 0, 1)))
    return G


def _advance(case, s, P, dt):
    law, g = case["law"], s.stencil
    axes = [a for a in range(3) if s.shape[a] > 1]
    U0 = U = _state(law, s.gamma, P, 0, "U")
    for b in {1: [1.0], 2: [1.0, 0.5], 3: [1.0, 0.25, 2.0 / 3]}[case["rk"]]:
        Q = _pad(P, s.bc, g)
        F = {}
        for a in axes:
            T = Q
            for t in axes:
                if t != a:  # one guard zone is kept across the faces
                    T = T.narrow(1 + t, g - 1, s.shape[t] + 2)
            L, R = _edges(T.movedim(1 + a, 1), case["recon"])
            F[a] = _riemann(law, case["riemann"], s.gamma, L, R, a).movedim(1, 1 + a)
        if law != "hydro":
            F = _ct(F, axes)
        dU = torch.zeros_like(U)
        for a in axes:
            f = F[a]
            for t in axes:
                if t != a:
                    f = f.narrow(1 + t, 1, s.shape[t])
            f = f.movedim(1 + a, 1)
            dU -= ((f[:, 1:] - f[:, :-1]) * (s.shape[a] / (s.upper[a] - s.lower[a]))).movedim(1, 1 + a)
        U = U0 * (1 - b) + (U + dt * dU) * b
        P = _recover(law, s.gamma, U, P)
    return P


def _exact_grid(case, s, seed, steps, t_final=None):
    P, t, dt = _interior(case, s, seed), 0.0, 0.0
    for _ in range(steps):
        dt = s.cfl * _courant(case, s, P)
        if t_final is not None:
            if t >= t_final:
                break
            dt = min(dt, t_final - t)
        P = _advance(case, s, P, dt)
        t += dt
    return _pad(P, s.bc, s.stencil).permute(1, 2, 3, 0).contiguous(), t, dt


def exact(case, seed):
    if case["kind"] == "batch":
        # the 2-D grids that need few steps
        got, times = [], []
        for k, s in enumerate(_grids(case)):
            fast = 1 / (_courant(case, s, _interior(case, s, 1000 * seed + k)) * s.cfl)
            if s.dims == 2 and 2 * fast * case["t_final"] < 60:
                got.append(_exact_grid(case, s, 1000 * seed + k, 1000, case["t_final"])[0])
            else:
                got.append(None)
            times.append(case["t_final"])
        return {"P": got, "t": np.array(times), "steps": None}
    P, t, dt = _exact_grid(case, _scheme(case), seed, case["steps"])
    return {"P": P, "dt": dt} if case["kind"] == "dropin" else {"P": P, "t": t}
