"""Performance cases of the AWCM framework: what a program that uses it spends its time in.

Each case is one call sequence through the public Python surface (package `awcm`, over the C-ABI):

  tube_step     one RK3 step of a 1D tube in the caller's own device buffers
                (awcm1d_step_noalloc): the smallest unit of work, latency alone counts
  tube_run      one 1D instance from its Riemann data, as one launch (AWCM1D.run)
  tube_batch    many 1D instances of uneven sizes, as one launch (AWCM1DBatch.run_all)
  advect_1d     the 1D scalar path (AWCM1DScalar.advance)
  euler_2d      a 2D Euler run from its initial state (AWCM2D.advance), any boundary manager
  advect_2d     the 2D scalar path (AWCM2DScalar.advance)
  gradient      loss and discrete adjoint of a frozen-mask run (AWCM2D.adjoint)
  flux          physical fluxes and spectral radii of device-resident states
                (euler_flux, euler_spectral_radius)

A solver's handle is kept between passes, as a program keeps it; a pass hands it the initial field
and masks, runs, and reads back the field and the masks.  Step counts are those of a short job, so
that the transfers weigh little, as they do in a full run (thousands of steps between two reads).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "c_pp-library_b200"))
import awcm  # noqa: E402
from awcm import _lib, gradient, workloads  # noqa: E402

BC = {"quadrants": awcm.BC_TRANSMISSIVE, "double_mach": awcm.BC_DOUBLE_MACH, "vortex": awcm.BC_PERIODIC,
      "shock_vortex": awcm.BC_SHOCK_VORTEX, "wind_tunnel": awcm.BC_WIND_TUNNEL}
PROBLEM = {"quadrants": awcm.PROBLEM_QUADRANTS, "double_mach": awcm.PROBLEM_DOUBLE_MACH,
           "vortex": awcm.PROBLEM_VORTEX, "shock_vortex": awcm.PROBLEM_SHOCK_VORTEX,
           "wind_tunnel": awcm.PROBLEM_WIND_TUNNEL}
DOMAIN = {"quadrants": (0.0, 1.0, 0.0, 1.0), "double_mach": (0.0, 4.0, 0.0, 1.0),
          "vortex": (0.0, 10.0, 0.0, 10.0), "shock_vortex": (-16.0, 8.0, -12.0, 12.0),
          "wind_tunnel": (0.0, 3.0, 0.0, 1.0)}


def listed():
    return [
        # The driver loop of a caller that owns its memory: one step of the Sod-sized tube (1025
        # points) in a developed flow.
        dict(name="tube_step_1025", kind="tube_step", levels=7, nx_coarse=17, scheme=awcm.WENOZ, tol=1e-4, warm=40),
        # The Sod benchmark: 1025 points, WENO-Z, whole run to t = 0.2 (about 900 steps).
        dict(name="tube_run_1025", kind="tube_run", levels=7, nx_coarse=17, scheme=awcm.WENOZ, tol=1e-4, t_end=0.2,
             steps=5000),
        # The shipped 1D driver's own grid and scheme: 16 coarse points, 11 levels (15361 points),
        # WENO5, threshold 1e-6: the largest line, with a coarse grid that is not a power of two.
        dict(name="tube_run_15361", kind="tube_run", levels=11, nx_coarse=16, scheme=awcm.WENO5, tol=1e-6, t_end=0.2,
             steps=300),
        # The uneven batch of the benchmark: 512 tubes of 257 to 8193 points, its opening steps.
        dict(name="tube_batch_512", kind="tube_batch", count=512, jmin=8, jmax=13, tol=1e-4, t_end=0.15, steps=200),
        # A small parameter study run to its end: fewer tubes than SMs, the longest one decides.
        dict(name="tube_batch_40", kind="tube_batch", count=40, jmin=8, jmax=11, tol=1e-4, t_end=0.04, steps=100000),
        # The 1D scalar driver's configuration: 13 levels on 9 coarse points (32769 points).
        dict(name="advect_1d_32769", kind="advect_1d", levels=13, nx_coarse=9, tol=1e-6, steps=100),
        # A small 2D job, 129 x 129: launches and latency.
        dict(name="quadrants_129", kind="euler_2d", problem="quadrants", levels=4, nxc=17, nyc=17, cfl=0.4, tol=1e-3,
             steps=100),
        # The headline workload: four quadrants on 2049 x 2049.
        dict(name="quadrants_2049", kind="euler_2d", problem="quadrants", levels=8, nxc=17, nyc=17, cfl=0.4, tol=1e-3,
             steps=600),
        # Double Mach reflection on a 4:1 grid, 2049 x 513, time-dependent boundary.
        dict(name="double_mach_2049x513", kind="euler_2d", problem="double_mach", levels=6, nxc=65, nyc=17, cfl=0.5,
             tol=1e-3, steps=300),
        # Smooth periodic flow on a ragged coarse grid (11 x 7 coarse points: 641 x 385).
        dict(name="vortex_641x385", kind="euler_2d", problem="vortex", levels=7, nxc=11, nyc=7, cfl=0.4, tol=1e-4,
             steps=200),
        # The 2D scalar path, 8 levels on 9 x 9 coarse points: 1025 x 1025.
        dict(name="advect_2d_1025", kind="advect_2d", levels=8, nxc=9, tol=1e-4, steps=200),
        # The gradient configuration: 513 x 513, periodic vortex with density bumps, 100 frozen steps
        # forward and the reverse sweep with sqrt(n) checkpoints, differentiable WENO-Z.
        dict(name="gradient_513", kind="gradient", levels=6, nxc=17, tol=1e-3, steps=100, every=0),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def line(nx_max):  # a dyadic 1D grid of up to nx_max points
        while True:
            levels, nxc = rng.randint(4, 11), rng.randint(9, 33)
            if 129 <= (nxc - 1) * 2 ** (levels - 1) + 1 <= nx_max:
                return dict(levels=levels, nx_coarse=nxc)

    kind = rng.choice(["tube_step", "tube_run", "tube_batch", "advect_1d", "euler_2d", "euler_2d", "euler_2d",
                       "advect_2d", "gradient", "flux"])
    if kind == "tube_step":
        return dict(kind=kind, **line(8193), scheme=rng.choice([awcm.WENOZ, awcm.WENO5]),
                    tol=rng.choice([1e-3, 1e-4, 1e-5]), warm=rng.randint(3, 80))
    if kind == "tube_run":
        return dict(kind=kind, **line(16385), scheme=rng.choice([awcm.WENOZ, awcm.WENO5]),
                    tol=rng.choice([1e-3, 1e-4, 1e-5]), t_end=0.2, steps=log_int(20, 600))
    if kind == "tube_batch":
        jmin = rng.randint(7, 10)
        return dict(kind=kind, count=log_int(2, 400), jmin=jmin, jmax=rng.randint(jmin, 13),
                    tol=rng.choice([1e-3, 1e-4]), t_end=0.15, steps=log_int(20, 200))
    if kind == "advect_1d":
        return dict(kind=kind, **line(32769), tol=rng.choice([1e-4, 1e-5, 1e-6]), steps=log_int(20, 200))
    if kind == "flux":
        return dict(kind=kind, n=log_int(1, 1 << 22), dim=rng.choice([1, 2, 2]))
    if kind == "gradient":
        levels = rng.randint(4, 6)
        return dict(kind=kind, levels=levels, nxc=rng.randint(9, 17), tol=rng.choice([1e-3, 1e-4]),
                    steps=log_int(4, 80), every=rng.choice([0, 0, 3, 1000]))
    while True:
        levels, nxc, nyc = rng.randint(4, 8), rng.randint(7, 65), rng.randint(7, 33)
        if kind == "advect_2d":
            nyc = nxc
        points = ((nxc - 1) * 2 ** (levels - 1) + 1) * ((nyc - 1) * 2 ** (levels - 1) + 1)
        if 4000 <= points <= 1500000:
            break
    if kind == "advect_2d":
        return dict(kind=kind, levels=levels, nxc=nxc, tol=rng.choice([1e-3, 1e-4]), steps=log_int(20, 200))
    return dict(kind=kind, problem=rng.choice(sorted(BC)), levels=levels, nxc=nxc, nyc=nyc, cfl=0.4,
                tol=rng.choice([1e-3, 1e-4]), steps=log_int(20, 200))


# ------------------------------------------------------------------------------------- inputs
def points(case, coarse="nx_coarse"):
    return (case[coarse] - 1) * 2 ** (case["levels"] - 1) + 1


def sod_like(case, rng):
    """Node range, interface and (rho, u, p) states of a shock tube near the Sod problem."""
    nx = points(case)
    s = rng.uniform(0.95, 1.05, 4)
    return (0.5 / nx, 1 - 0.5 / nx), rng.uniform(0.48, 0.52), (1.0 * s[0], 0.0, 1.0 * s[1]), (
        0.125 * s[2], 0.0, 0.1 * s[3])


def pulse(x, rng):
    """Advected field of the scalar paths: a Gaussian and a step, centred by the seed (one axis)."""
    c = rng.uniform(-0.1, 0.1)
    return np.exp(-200.0 * (x - c) ** 2) + (np.abs(x - c - 0.25) < 0.05)


def new_masks(planes, shape):
    """The masks a new instance starts with: mask0 set everywhere, the others clear."""
    m = np.zeros((planes,) + shape, np.uint8)
    m[1] = 1
    return m


def prepare(case, seed):
    rng = np.random.default_rng([20261205, seed])
    kind = case["kind"]
    s = dict(case=case)
    if kind == "tube_step":
        (x0, x1), xi, left, right = sod_like(case, rng)
        b = awcm.AWCM1D(case["levels"], case["nx_coarse"], x0, x1, scheme=case["scheme"])
        b.init_riemann(xi, left, right)
        w = b.nx + 6
        state = np.full(5 * w, 0, np.uint8)
        state[:w] = 0x01
        state[:3] = state[w - 3:w] = 0xE1
        s["geometry"] = (case["levels"], case["nx_coarse"], x0, x1, 1.4, case["scheme"], case["tol"], 0.5)
        s["q"] = torch.from_numpy(np.ascontiguousarray(b.get_q().T)).cuda()
        s["state"] = torch.from_numpy(state).cuda()
        s["out"] = torch.zeros(16, dtype=torch.float64, device="cuda")
        for _ in range(case["warm"]):
            tube_step(s)
        s["q0"], s["state0"] = s["q"].clone(), s["state"].clone()
    elif kind == "tube_run":
        (x0, x1), xi, left, right = sod_like(case, rng)
        b = awcm.AWCM1D(case["levels"], case["nx_coarse"], x0, x1, scheme=case["scheme"])
        b.init_riemann(xi, left, right)
        s |= dict(solver=b, q0=b.get_q(), m0=new_masks(5, (b.nx + 6,)))
    elif kind == "tube_batch":
        tubes = workloads.shock_tubes(case["count"], seed=int(rng.integers(1 << 31)), jmax=(case["jmin"], case["jmax"]))
        # every seed and every half of the list has the whole range of sizes: the work is alike
        for k, t in enumerate(tubes):
            J = case["jmin"] + k % (case["jmax"] - case["jmin"] + 1)
            nx = 2 ** J + 1
            t |= dict(jmax=J, num_levels=J - 3, nx=nx, x_min=0.5 / nx, x_max=1 - 0.5 / nx)
        b = workloads.make_batch(awcm, tubes)
        s |= dict(solver=b, q0=[b.get_q(k) for k in range(b.n)], m0=[new_masks(5, (nx + 6,)) for nx in b.nx])
    elif kind == "advect_1d":
        b = awcm.AWCM1DScalar([case["levels"]], case["nx_coarse"], -0.5, 0.5)
        nx = b.nx[0]
        x = -0.5 + (np.arange(nx + 6) - 3) / (nx - 1)
        s |= dict(solver=b, q0=pulse(x, rng), m0=new_masks(5, (nx + 6,)), dt=0.5 / (nx - 1))
    elif kind == "advect_2d":
        n = points(case, "nxc")
        d = 1.0 / n
        b = awcm.AWCM2DScalar(case["levels"], case["nxc"], case["nxc"], 0.5 * d, 1 - 0.5 * d, 0.5 * d, 1 - 0.5 * d)
        x = 0.5 * d + (np.arange(n + 6) - 3) * d
        cx, cy = rng.uniform(0.45, 0.55, 2)
        s |= dict(solver=b, q0=np.exp(-50 * (x[None, :] - cx) ** 2 - 50 * (x[:, None] - cy) ** 2), dt=0.4 * d)
    elif kind == "euler_2d":
        p = case["problem"]
        b = awcm.AWCM2D(case["levels"], case["nxc"], case["nyc"], *DOMAIN[p], BC[p])
        u, v = rng.uniform(-1, 1, 2)
        at = {"quadrants": (0.5 + 0.05 * u, 0.5 + 0.05 * v), "double_mach": (1.4 + 0.05 * u, 0.0),
              "vortex": (5 + u, 5 + v), "shock_vortex": (2 + 0.2 * u, 0.2 * v), "wind_tunnel": (0.0, 0.0)}[p]
        b.init_problem(PROBLEM[p], *at)
        q0 = b.get_q()
        if p == "wind_tunnel":  # a uniform start has one state only: scale the gas by the seed
            q0 *= 1 + 0.05 * u
        s |= dict(solver=b, q0=q0, m0=new_masks(5, (b.ny + 6, b.nx + 6)))
    elif kind == "gradient":
        b = awcm.AWCM2D(case["levels"], case["nxc"], case["nxc"], 0.0, 10.0, 0.0, 10.0, awcm.BC_PERIODIC)
        base = int(rng.integers(1 << 31))
        q0, target = gradient.vortex_bumps(b, base), gradient.target_density(b, base + 1)
        b.set_q(q0)
        b.prepare(case["tol"])
        b.set_wenoz(1e-6, 1e-6)
        s |= dict(solver=b, q0=b.get_q(), target=target, dt=gradient.stable_dt(q0, 10.0 / (b.nx - 1)))
    else:
        n, dim = case["n"], case["dim"]
        rho, pr = 10.0 ** rng.uniform(-1, 1, (2, n))
        vel = rng.uniform(-1, 1, (dim, n))
        q = np.stack([rho, *(rho * vel), pr / 0.4 + 0.5 * rho * (vel * vel).sum(0)], axis=1)
        s["q"] = torch.from_numpy(q).cuda()
        s["flux"] = [torch.empty_like(s["q"]) for _ in range(dim)]
        s["speed"] = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(dim)]
    return s


# ---------------------------------------------------------------------------------------- runs
def tube_step(s):
    _lib.call("awcm1d_step_noalloc", *s["geometry"], 0.0, 1.0, s["q"].data_ptr(), s["state"].data_ptr(),
              s["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)


def run(state):
    s, case = state, state["case"]
    kind, b = case["kind"], state.get("solver")
    if kind == "tube_step":
        s["q"].copy_(s["q0"])
        s["state"].copy_(s["state0"])
        tube_step(s)
        w = s["q"].shape[1]
        return dict(q=s["q"], masks=s["state"][:w] & 0x1F, levels=s["state"][w:], out=s["out"])
    if kind == "tube_run":
        b.set_q(s["q0"])
        b.set_masks(s["m0"])
        _, t, _ = b.run(case["tol"], 0.5, case["t_end"], case["steps"])
        return dict(q=b.get_q(), masks=b.get_masks(), t=t)
    if kind == "tube_batch":
        for k in range(b.n):
            b.set_q(k, s["q0"][k])
            b.set_masks(k, s["m0"][k])
        b.set_run(case["tol"], 0.5, 0.0, case["t_end"])
        b.run_all(case["steps"])
        b.sync()
        return dict(q=np.concatenate([b.get_q(k) for k in range(b.n)]),
                    masks=np.concatenate([b.get_masks(k) for k in range(b.n)], axis=1))
    if kind == "advect_1d":
        b.set_q(0, s["q0"])
        b.b.set_masks(0, s["m0"])
        b.advance(case["tol"], s["dt"], case["steps"])
        return dict(q=b.get_q(0), masks=b.get_masks(0))
    if kind == "advect_2d":
        b.set_q(s["q0"])
        t, steps, points_done = b.advance(case["tol"], s["dt"], 0.0, case["steps"])
        return dict(q=b.get_q(), masks=b.get_masks(), t=t)
    if kind == "euler_2d":
        b.set_q(s["q0"])
        b.set_masks(s["m0"])
        t, steps, points_done, stage_points = b.advance(case["tol"], case["cfl"], 0.0, 1e9, case["steps"])
        return dict(q=b.get_q(), masks=b.get_masks(), t=t, steps=steps, points=int(points_done))
    if kind == "gradient":
        b.set_q(s["q0"])
        loss, grad, _ = b.adjoint(0.0, s["dt"], case["steps"], s["target"], case["every"])
        return dict(loss=loss, grad=grad)
    n, dim = case["n"], case["dim"]
    stream = torch.cuda.current_stream().cuda_stream
    for d in range(dim):
        awcm.euler_flux(s["q"].data_ptr(), s["flux"][d].data_ptr(), n, dim, d, 1.4, stream)
        awcm.euler_spectral_radius(s["q"].data_ptr(), s["speed"][d].data_ptr(), n, dim, d, 1.4, stream)
    return dict(flux=s["flux"], speed=s["speed"])


# ---------------------------------------------------------------------------------------- work
# Operations of the reference's face flux and coarse derivative (adds, multiplies, divisions, roots).
FACE_1D, FACE_2D, FACE_SCALAR, COARSE = 1007, 1354, 90, 110


def work(case):
    """Bytes and operations of one pass.  The active set is found by the run itself: the counts
    below are typical ones (points of mask0 per step; faces of the three stages are about six
    times that in one dimension and ten in two)."""
    kind = case["kind"]
    steps = case.get("steps", 1)
    if kind == "flux":
        n, d = case["n"], case["dim"]
        c = d + 2
        return dict(bytes=8.0 * n * (c + d * (c + 1)), flops=n * d * (6.0 * c + 12))
    if kind in ("tube_step", "tube_run"):
        nx = points(case)
        active = min(nx, 60 + 16 * case["levels"])
        if kind == "tube_run" and case["levels"] == 7:
            steps = min(steps, 900)
        return dict(bytes=2.0 * nx * (24 + 5) + steps * 2 * 24.0 * active, flops=steps * active * 3.0 * FACE_1D)
    if kind == "tube_batch":
        total = dict(bytes=0.0, flops=0.0)
        for k in range(case["count"]):
            J = case["jmin"] + k % (case["jmax"] - case["jmin"] + 1)
            nx, active = 2 ** J + 1, 60 + 16 * (J - 3)
            n = min(steps, case["t_end"] * nx * 4)
            total["bytes"] += 2.0 * nx * (24 + 5) + n * 2 * 24.0 * active
            total["flops"] += n * active * 3.0 * FACE_1D
        return total
    if kind == "advect_1d":
        nx = points(case)
        active = min(nx, 40 * case["levels"])
        return dict(bytes=2.0 * nx * 13 + steps * 2 * 8.0 * active, flops=steps * active * 3.0 * FACE_SCALAR)
    nx = points(case, "nxc")
    ny = points(case, "nyc") if "nyc" in case else nx
    active = min(nx * ny, 25 * (nx + ny))
    if kind == "advect_2d":
        return dict(bytes=2.0 * nx * ny * 13 + steps * 2 * 8.0 * active, flops=steps * active * 6.0 * FACE_SCALAR)
    if kind == "euler_2d":
        return dict(bytes=2.0 * nx * ny * 37 + steps * 2 * 32.0 * active, flops=steps * active * 6.0 * FACE_2D)
    # forward once, recomputed once, and the reverse of each face at about three times its cost
    return dict(bytes=2.0 * nx * ny * 32 + nx * ny * 8 + steps * 8 * 32.0 * active,
                flops=steps * active * 5 * 6.0 * FACE_2D)


# --------------------------------------------------------------------------------------- exact
class Line:
    """A 1D AWCM instance in plain numpy, 64 bits: fields of nx + 6 values (three ghosts a side)."""

    def __init__(self, levels, nx_coarse, x0, x1, scheme):
        self.maxl, self.scheme = levels - 1, scheme
        self.nx = (nx_coarse - 1) * 2 ** (levels - 1) + 1
        self.n1, self.w = self.nx - 1, self.nx + 6
        self.dx = (x1 - x0) / (self.nx - 1)
        self.mask = np.zeros((4, self.w), bool)
        self.mask[0] = True
        self.temp = np.zeros(self.w, bool)
        self.level = np.zeros((4, self.w), int)
        self.weight = np.ones((4, 5))
        for j in range(-1, 4):
            for i in range(4):
                for k in range(4):
                    if k != i:
                        self.weight[i, j + 1] *= (j + 0.5 - k) / (i - k)

    def details(self, lev):
        """Detail points of a level, their four coarse neighbours and weights (as array indices)."""
        D = 1 << (self.maxl - lev)
        h = D >> 1
        i = h + D * np.arange(self.n1 // D)
        first, side = i - D - h, np.ones(len(i), int)
        lo, hi = first < 0, i + D + h > self.n1
        first[lo], side[lo] = 0, 0
        hi &= ~lo
        first[hi], side[hi] = self.n1 - 3 * D, 2
        return i + 3, first[None] + 3 + D * np.arange(4)[:, None], self.weight[:, side + 1]

    def evens(self, lev):
        """Interior coarse points of a level, their four detail neighbours and weights."""
        D = 1 << (self.maxl - lev)
        h = D >> 1
        i = D + D * np.arange(self.n1 // D - 1)
        first, side = i - D - h, np.ones(len(i), int)
        lo, hi = first < 0, i + D + h > self.n1
        first[lo], side[lo] = h, 0
        hi &= ~lo
        first[hi], side[hi] = self.n1 - 3 * D - h, 2
        return i + 3, first[None] + 3 + D * np.arange(4)[:, None], self.weight[:, side + 1]

    def forward(self, q, tol):
        m = self.mask[0]
        for lev in range(self.maxl - 1, -1, -1):
            i, at, wt = self.details(lev)
            v = q[i].copy()
            for c in range(4):
                v = v - wt[c] * q[at[c]]
            v *= 0.5
            on = m[i]
            q[i[on]] = v[on]
            m[i[on & (np.abs(v) < tol)]] = False
            i, at, wt = self.evens(lev)
            v = q[i].copy()
            for c in range(4):
                v = v + wt[c] * q[at[c]]
            on = m[i]
            q[i[on]] = v[on]

    def inverse(self, q, m):
        for lev in range(self.maxl):
            i, at, wt = self.evens(lev)
            v = q[i].copy()
            for c in range(4):
                v = v - wt[c] * q[at[c]]
            q[i] = np.where(m[i], v, 0.0)
            i, at, wt = self.details(lev)
            v = q[i] * 2
            for c in range(4):
                v = v + wt[c] * q[at[c]]
            q[i] = np.where(m[i], v, 0.0)

    def close(self, m):
        for lev in range(self.maxl - 1, -1, -1):
            i, at, _ = self.details(lev)
            m[at[:, m[i]].ravel()] = True

    def adjacent(self, m, source):
        i = np.arange(1, self.n1)
        low = i & -i
        i, low = i[(low < (1 << self.maxl)) & source[3 + i]], low[(low < (1 << self.maxl)) & source[3 + i]]
        off = np.maximum(low // 2, 1)
        m[i - off + 3] = True
        m[i + off + 3] = True

    def levels(self, k):
        m, out = self.mask[k], self.level[k]
        i = np.arange(self.nx)
        seen = np.zeros(self.nx, bool)
        found = np.where(m[3:-3], out[3:-3], 0)
        for lev in range(self.maxl, -1, -1):
            d = 1 << (self.maxl - lev)
            a, b = i - d, i + d
            near = np.where(a < -3, True, m[np.maximum(a, -3) + 3]) | np.where(
                b > self.n1 + 3, True, m[np.minimum(b, self.n1 + 3) + 3])
            new = near & ~seen & m[3:-3]
            found[new] = lev
            seen |= new
        found[0] = found[-1] = self.maxl
        out[3:-3] = found

    def stencils(self, m, source, level):
        i = np.nonzero(source[3:-3])[0]
        lev = level[3 + i]
        fine = i[lev == self.maxl]
        for c in range(-3, 4):
            m[fine + c + 3] = True
        i, d = i[lev != self.maxl], 1 << (self.maxl - lev[lev != self.maxl])
        first, sign, count = i - 2 * d, np.ones(len(i), int), np.full(len(i), 5)
        left, right = i - 2 * d <= 0, (i - 2 * d > 0) & (i + 2 * d >= self.n1)
        first[left], first[right], sign[right] = 0, self.n1, -1
        count[left | right] = 6
        for c in range(6):
            x = first + sign * c * d
            x = x[(c < count) & (x >= -3) & (x <= self.n1 + 3)]
            m[x + 3] = True

    def adapt(self, q, tol):
        """PrepareEuler, or Prepare of the scalar path."""
        scalar = self.scheme == awcm.SCALAR_ADVECTION
        m = self.mask
        if not scalar:
            self.temp = m[0].copy()
        self.forward(q[0], tol)
        m[0, 3:6] = m[0, -6:-4] = True
        m[0, -4] = True
        self.adjacent(m[0], m[0].copy())
        self.close(m[0])
        for k in (1, 2, 3):
            self.levels(k - 1)
            m[k] = m[k - 1]
            if not scalar:
                self.adjacent(m[k], m[k - 1])
            self.stencils(m[k], m[k].copy(), self.level[k - 1])
            self.close(m[k])
        self.levels(3)
        self.inverse(q[0], m[3])
        if scalar:
            return
        new = m[3] & ~self.temp
        new[:3] = new[-3:] = False
        self.close(new)
        for lev in range(self.maxl):
            i, at, wt = self.details(lev)
            on = new[i] & ~self.temp[i]
            for p in (1, 2):
                v = np.zeros(len(i))
                for c in range(4):
                    v = v + wt[c] * q[p][at[c]]
                q[p][i[on]] = v[on]

    def edges(self, q):
        for x in q:
            x[:3], x[-3:] = x[3], x[-4]

    def sound(self, q):
        return np.sqrt(1.4 * (0.4 * (q[2] - 0.5 * (q[1] * q[1]) / q[0])) / q[0])

    def speed(self, q, on):
        a = q[:, 3:-3][:, on]
        return float(np.max(np.abs(a[1] / a[0]) + self.sound(a), initial=0.0))

    def step(self, q, tol, cfl, t, t_end):
        """One RK3 step of the Euler path; q: three fields, in place.  Returns dt."""
        self.adapt(q, tol)
        dt = cfl * self.dx / self.speed(q, self.mask[3, 3:-3])
        dt = t_end - t if t + dt > t_end else dt
        start = None
        for stage, k in enumerate((2, 1, 0)):
            self.edges(q)
            fast = k + 1
            alpha = self.speed(q, self.mask[fast, 3:-3] & (self.level[fast, 3:-3] == self.maxl))
            start = q.copy() if stage == 0 else start
            on = np.nonzero(self.mask[k, 3:-3])[0]
            d = 1 << (self.maxl - self.level[k, 3 + on])
            on, d = on[(d == 1) | ((on - 2 * d >= -3) & (on + 2 * d <= self.n1 + 3))], d[
                (d == 1) | ((on - 2 * d >= -3) & (on + 2 * d <= self.n1 + 3))]
            dF = self.differences(q, on, d, alpha)
            i = on + 3
            r = q[:, i] - dt / (self.dx * d) * dF
            q[:, i] = r if stage == 0 else 0.75 * start[:, i] + 0.25 * r if stage == 1 else (
                start[:, i] + 2.0 * r) / 3.0
        q[:, 3:-3][:, ~self.mask[0, 3:-3]] = 0
        return dt

    def flux(self, q):
        u, p = q[1] / q[0], 0.4 * (q[2] - 0.5 * (q[1] * q[1]) / q[0])
        return np.stack([q[0] * u, q[0] * u * u + p, (q[2] + p) * u])

    def differences(self, q, on, d, alpha):
        out = np.zeros((3, len(on)))
        fine = d == 1
        f = np.unique(np.concatenate([on[fine] - 1, on[fine]]))  # face f + 1/2
        face = np.zeros((3, self.nx + 1))
        if len(f):
            face[:, f + 1] = self.faces(q[:, f[None] + 1 + np.arange(6)[:, None]], alpha)
        out[:, fine] = face[:, on[fine] + 1] - face[:, on[fine]]
        one, two = (2 / 3, -1 / 12), (1 / 12, -2 / 3, 0.0, 2 / 3, -1 / 12)
        edge = (-1 / 3, -0.5, 1.0, -1 / 6)
        n = self.n1
        for sel, sign, at, wt in (
                (on - 2 * d < 0, 1, (-1, 0, 1, 2), edge), (on == 2 * d, 1, (-2, -1, 0, 1, 2), two),
                (on > n - 2 * d, -1, (-1, 0, 1, 2), edge), (on + 2 * d == n, -1, (-2, -1, 0, 1, 2), two)):
            sel = sel & ~fine & (out == 0).all(0)
            out[:, sel] = sum(c * self.flux(q[:, on[sel] + sign * a * d[sel] + 3]) for a, c in zip(at, wt))
        sel = ~fine & (on - 2 * d > 0) & (on + 2 * d < n)
        F = [self.flux(q[:, on[sel] + a * d[sel] + 3]) for a in (-2, -1, 1, 2)]
        out[:, sel] = one[0] * (F[2] - F[1]) + one[1] * (F[3] - F[0])
        return out

    def faces(self, s, alpha):
        """Characteristic Lax-Friedrichs face flux; s: three components of six cells of each face."""
        l, r = s[:, 2], s[:, 3]
        wide = [(c[2] + 0.4 * (c[2] - 0.5 * (c[1] * c[1]) / c[0])) / c[0] for c in (l, r)]
        a, b = np.sqrt(l[0]), np.sqrt(r[0])
        u = (a * (l[1] / l[0]) + b * (r[1] / r[0])) / (a + b)
        H = (a * wide[0] + b * wide[1]) / (a + b)
        c = np.sqrt(0.4 * (H - 0.5 * u * u))

        def waves(x):
            x2 = ((H - u * u) * x[0] + u * x[1] - x[2]) * (0.4 / (c * c))
            x3 = (x[1] + (c - u) * x[0] - c * x2) / (2 * c)
            return np.stack([x[0] - x2 - x3, x2, x3])

        q, f = waves(s), waves(self.flux(s))
        up, down = 0.5 * (f + alpha * q), 0.5 * (f - alpha * q)
        S = self.upwind(up[:, 4], up[:, 3], up[:, 2], up[:, 1], up[:, 0]) + self.upwind(
            down[:, 1], down[:, 2], down[:, 3], down[:, 4], down[:, 5])
        first = (np.ones_like(u), np.ones_like(u), np.ones_like(u))
        second = (u - c, u, u + c)
        third = (H - u * c, 0.5 * (u * u), H + u * c)
        return np.stack([S[0] * x[0] + S[1] * x[1] + S[2] * x[2] for x in (first, second, third)])

    def upwind(self, ll, l, c, r, rr):
        b = (13 / 12 * (c - 2 * r + rr) ** 2 + 0.25 * (3 * c - 4 * r + rr) ** 2,
             13 / 12 * (l - 2 * c + r) ** 2 + 0.25 * (l - r) ** 2,
             13 / 12 * (ll - 2 * l + c) ** 2 + 0.25 * (ll - 4 * l + 3 * c) ** 2)
        if self.scheme == awcm.WENOZ:
            tau = np.abs(b[0] - b[2])
            a = [d * (1 + tau / (x + 1e-40)) for d, x in zip((0.1, 0.6, 0.3), b)]
        else:
            a = [d / ((1e-6 + x) * (1e-6 + x)) for d, x in zip((0.1, 0.6, 0.3), b)]
        total = a[0] + a[1] + a[2]
        return (a[0] / total * (11 / 6 * c + -7 / 6 * r + 1 / 3 * rr) + a[1] / total * (1 / 3 * l + 5 / 6 * c - 1 / 6 * r)
                + a[2] / total * (-1 / 6 * ll + 5 / 6 * l + 1 / 3 * c))

    def packed(self):
        """The masks as the allocation-free step keeps them: a byte a point."""
        return (sum(self.mask[k].astype(np.uint8) << k for k in range(4)) | (self.temp.astype(np.uint8) << 4)).astype(
            np.uint8)


def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng([20261205, seed])
    if kind == "flux":
        q = prepare(case, seed)["q"]
        dim = case["dim"]
        vel = q[:, 1:-1] / q[:, :1]
        p = 0.4 * (q[:, -1] - 0.5 * (q[:, 1:-1] ** 2).sum(1) / q[:, 0])
        c = torch.sqrt(1.4 * p / q[:, 0])
        flux = []
        for d in range(dim):
            f = q * vel[:, d:d + 1]
            f[:, 1 + d] += p
            f[:, -1] += p * vel[:, d]
            flux.append(f)
        return dict(flux=flux, speed=[vel[:, d].abs() + c for d in range(dim)])
    if kind in ("tube_step", "tube_run") and case.get("steps", 1) * points(case) <= 6e6:
        (x0, x1), xi, left, right = sod_like(case, rng)
        o = Line(case["levels"], case["nx_coarse"], x0, x1, case["scheme"])
        x = x0 + o.dx * (np.arange(o.w) - 3)
        rho, u, p = (np.where(x <= xi, a, b) for a, b in zip(left, right))
        q = np.stack([rho, rho * u, p / 0.4 + 0.5 * rho * (u * u)])
        if kind == "tube_step":
            for _ in range(case["warm"] + 1):
                o.step(q, case["tol"], 0.5, 0.0, 1.0)
            return dict(q=q, masks=None, levels=None, out=None)
        t, steps = 0.0, 0
        while t < case["t_end"] and steps < case["steps"]:
            t += o.step(q, case["tol"], 0.5, t, case["t_end"])
            steps += 1
        return dict(q=np.ascontiguousarray(q.T), masks=None, t=t)
    # A batch, a 2D run or an adjoint: the same arithmetic over millions of points and hundreds of
    # steps takes plain numpy far longer than the 20 seconds an exact value may take.
    return None
