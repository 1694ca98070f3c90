"""The work that programs give this library, as cases that can be timed and compared.

A suspension program does the same few things over and over: it applies the mobility
(spread, Stokes solve, interpolation) of its blobs at fixed positions for one force
after another (every GMRES iteration does), it moves the blobs and applies it there,
it draws the fluctuating field, it solves the rigid-body saddle-point system, and it
takes whole time steps of one suspension or of an ensemble.  Each case is one of these
through the public Python interface (``fcm.py``), with device arrays where a program
keeps them there.

``listed`` gives the cases, ``draw`` another one of the same ranges, ``prepare`` the
inputs and the context that a program keeps, ``run`` one pass, ``work`` the bytes and
operations a pass cannot do without, ``exact`` the result in plain 64-bit torch.

Velocities of the FP32 grid are handed over as float32, the accuracy they have; the
interface returns them widened to FP64.
"""
import functools
import math

import numpy as np
import torch

from timstochrigidbodiessim_b200 import configs
from timstochrigidbodiessim_b200.fcm import Suspension, step_many
from timstochrigidbodiessim_b200.params import FcmParams, rod_reference_positions

MIXED_TOL = 1e-8  # refinement tolerance of mixed-precision solves (FP64 ones solve to 1e-10)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest suspension, moved and applied once: 32 rods, 64^3 grid, FP64 (launch latency)
        dict(name="mobility64_rods32_g64", kind="mobility", precision=0, fresh=True, bodies=32, blobs=6,
             nx=64, ny=64, nz=64, dx=1.0, tuned=False),
        # 2048 rods at volume fraction 0.10, the ordinary FP64 suspension, at new positions
        dict(name="mobility64_rods2048_g256", kind="mobility", precision=0, fresh=True, bodies=2048, blobs=6,
             nx=256, ny=256, nz=256, dx=0.3130521124285032, tuned=False),
        # 32,768 random clusters at volume fraction 0.20, FP64: one residual product of the largest suspension
        dict(name="mobility64_clusters32768_g512", kind="mobility", precision=0, fresh=False, bodies=32768, blobs=12,
             nx=512, ny=512, nz=512, dx=0.3943, tuned=False),
        # a box whose sides are neither equal nor multiples of the 8-point tile
        dict(name="mobility64_box_100x126x90", kind="mobility", precision=0, fresh=True, bodies=250, blobs=6,
             nx=100, ny=126, nz=90, dx=0.45, tuned=False),
        # an ensemble member's FP32 product (one GMRES iteration of a small suspension)
        dict(name="mobility32_rods300_g96", kind="mobility", precision=1, fresh=False, bodies=300, blobs=6,
             nx=96, ny=96, nz=96, dx=0.45, tuned=False),
        # the ordinary suspension's FP32 product
        dict(name="mobility32_rods2048_g256", kind="mobility", precision=1, fresh=False, bodies=2048, blobs=6,
             nx=256, ny=256, nz=256, dx=0.3130521124285032, tuned=False),
        # the largest suspension's FP32 product, with the kernels fcm_autotune chooses (as bench.py runs it)
        dict(name="mobility32_clusters32768_g512", kind="mobility", precision=1, fresh=False, bodies=32768, blobs=12,
             nx=512, ny=512, nz=512, dx=0.3943, tuned=True),
        # the fluctuating velocity field and its blob velocities, once per step, FP64
        dict(name="noise64_rods2048_g256", kind="noise", precision=0, bodies=2048, blobs=6,
             nx=256, ny=256, nz=256, dx=0.3130521124285032),
        # a whole FP64 GMRES solve of the CPU-sized suspension (host-driven, dozens of small launches an iteration)
        dict(name="solve64_rods32_g64", kind="solve", precision=0, bodies=32, blobs=6, grid=64, box=64.0),
        # an Euler-Maruyama step, mixed precision, device-resident, tuned: the production step
        dict(name="step_em_mixed_rods2048_g256", kind="step", algorithm=2, precision=1, channel=False, bodies=2048,
             blobs=6, grid=256, box=80.14134078169682, tuned=True),
        # a drifter-corrector step in the slip channel, FP64: the reference's default geometry and algorithm
        dict(name="step_gdc64_channel40_g96", kind="step", algorithm=1, precision=0, channel=True, bodies=40, blobs=6,
             grid=96, box=40.0, tuned=False),
        # eight members of the 64-suspension ensemble (50-500 rods, 64^3-96^3) stepped together, mixed precision
        dict(name="ensemble8_em_mixed", kind="ensemble", members=8, first=0, precision=1, tuned=True),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["mobility", "mobility", "mobility", "noise", "solve", "step", "ensemble"])
    if kind in ("mobility", "noise"):
        precision = rng.choice([0, 1]) if kind == "mobility" else 0
        unit = rng.choice([2, 8, 16, 32])  # any even sides, whole tiles, the transforms' usual lengths
        n = [max(32, unit * round(_log(rng, 32, 320) / unit)) for _ in range(3)]
        if rng.random() < 0.5:
            n = [n[0]] * 3
        while n[0] * n[1] * n[2] > 320 ** 3:
            n = [max(32, unit * (k // (2 * unit))) for k in n]
        dx, phi, blobs = round(rng.uniform(0.3, 0.6), 4), rng.uniform(0.03, 0.2), rng.choice([6, 12])
        vol = n[0] * n[1] * n[2] * dx ** 3
        bodies = max(1, min(16384, int(phi * vol / (blobs * 4.0 / 3.0 * math.pi))))
        c = dict(kind=kind, precision=precision, bodies=bodies, blobs=blobs, nx=n[0], ny=n[1], nz=n[2], dx=dx)
        if kind == "mobility":
            c.update(fresh=rng.random() < 0.5, tuned=precision == 1 and rng.random() < 0.5)
        return c
    if kind == "solve":
        grid = rng.choice([32, 48, 64, 72, 80, 96])
        return dict(kind=kind, precision=0, bodies=rng.randint(4, 30), blobs=rng.choice([4, 6]), grid=grid,
                    box=round(grid * rng.uniform(0.7, 1.0), 3))
    if kind == "step":
        channel = rng.random() < 0.3
        bodies, blobs = rng.randint(20, 60) if channel else int(_log(rng, 60, 600)), 6
        phi = rng.uniform(0.01, 0.025) if channel else rng.uniform(0.03, 0.1)
        box = round((bodies * blobs * 4.0 / 3.0 * math.pi / phi) ** (1.0 / 3.0), 3)
        return dict(kind=kind, algorithm=rng.choice([1, 2]), precision=rng.choice([0, 1]), channel=channel, bodies=bodies,
                    blobs=blobs, grid=configs.nearest_fft_size(box * rng.uniform(1.8, 2.6), lo=48, hi=128), box=box,
                    tuned=rng.random() < 0.5)
    precision = rng.choice([0, 1])
    return dict(kind=kind, members=rng.randint(2, 8 if precision == 1 else 4), first=rng.randint(8, 48),
                precision=precision, tuned=rng.random() < 0.5)


# ------------------------------------------------------------------ inputs
def _rotations(q):
    return torch.from_numpy(configs.rotation_matrices(q))


def _cloud(case, seed):
    """Blob positions (Nb, 3) of rods or compact clusters near the sites of a jittered lattice, and blob forces."""
    rng = np.random.default_rng(seed)
    M, nb = case["bodies"], case["blobs"]
    box = np.array([case["nx"], case["ny"], case["nz"]]) * case["dx"]
    if nb == 12:
        ref = configs.random_walk_cluster(rng, nb, draws=8)
    else:
        ref = np.array(rod_reference_positions(nb, 2.2)).reshape(-1, 3)
    sp = (box.prod() / M) ** (1.0 / 3.0)
    m = np.maximum(1, np.floor(box / sp)).astype(int)
    while m.prod() < M:
        m[np.argmin(m / box)] += 1
    site = rng.permutation(int(m.prod()))[:M]
    ijk = np.stack([site // (m[1] * m[2]), (site // m[2]) % m[1], site % m[2]], axis=1)
    x = (ijk + 0.5 + rng.uniform(-0.3, 0.3, (M, 3))) * (box / m)
    R = configs.rotation_matrices(configs.random_unit_quaternions(rng, M))
    Y = x[:, None, :] + np.einsum("nij,mj->nmi", R, ref)
    Y = (Y.reshape(-1, 3) % box) % box
    return ref, Y, rng.standard_normal(3 * M * nb)


@functools.lru_cache(maxsize=32)
def _placed(channel, bodies, blobs, grid, box):
    """A suspension of non-overlapping rods, the same for every seed (_moved makes them differ)."""
    if channel:
        return configs.rod_channel(bodies, grid, box, nb=blobs, seed=7)
    return configs.rod_suspension(bodies, grid, L=box, nb=blobs, seed=7)


@functools.lru_cache(maxsize=64)
def _member(i):
    d, ref, x, q, fe = configs.ensemble_member(i)
    return FcmParams.defaults(**d), ref, x, q, fe


def _moved(rng, p, x):
    """The bodies shifted together through the periodic box (along the walls in a channel)."""
    L = np.array(p.box)
    shift = rng.uniform(0.0, 1.0, 3) * L * np.array([1.0, 0.0 if p.slip_channel else 1.0, 1.0])
    return ((x.reshape(-1, 3) + shift) % L % L).ravel()


def _context(p, ref, x, q, fe, stream, tuned):
    s = Suspension(p, ref, stream=stream)
    s.set_bodies(x, q)
    s.set_external_forces(fe)
    s.produce_reference_matrices()
    if tuned:
        s.fill_all_blob_pos()
        s.set_up_gaussians()
        s.autotune(reps=3)
    return s


def _stepped(p0, ref, x0, q0, fe, case, seed, stream):
    """A running simulation: its context, one step behind it, and the bodies of the step to come."""
    rng = np.random.default_rng(seed)
    p = p0.copy(algorithm=case.get("algorithm", 2), precision=case["precision"], noise=1)
    if p.precision == 1:
        p.gmres_tol = MIXED_TOL
    x = _moved(rng, p, x0)
    s = _context(p, ref, x, q0, fe, stream, case["tuned"])
    s.step_async(seed, 0)
    s.step_wait()
    return dict(s=s, x=torch.from_numpy(x).cuda(), q=torch.from_numpy(np.ascontiguousarray(q0)).cuda(), seed=seed)


def _solve_inputs(case, seed):
    p, ref, x0, q, fe = _placed(False, case["bodies"], case["blobs"], case["grid"], case["box"])
    rng = np.random.default_rng(seed)
    x = _moved(rng, p, x0)
    V, F = rng.standard_normal(3 * p.num_blobs), rng.standard_normal(3 * p.num_blobs)
    return p, ref, x, q, fe, V, F


def prepare(case, seed):
    kind, stream = case["kind"], torch.cuda.current_stream()
    if kind in ("mobility", "noise"):
        ref, Y, F = _cloud(case, seed)
        L = case["dx"] * min(case["nx"], case["ny"], case["nz"])
        p = FcmParams.defaults(nx=case["nx"], ny=case["ny"], nz=case["nz"], ngauss=20, dx=case["dx"],
                               num_bodies=case["bodies"], blobs_per_body=case["blobs"], ncells=max(3, int(L // 2.2)),
                               potential=3, gmres_max_iter=100, gmres_tol=1e-10, dt=0.01, precision=case["precision"])
        s = Suspension(p, ref.ravel(), stream=stream)
        Y, F = torch.from_numpy(Y.ravel()).cuda(), torch.from_numpy(F).cuda()
        s.set_up_gaussians(Y)
        if case.get("tuned"):
            s.autotune(reps=3)
        return dict(case=case, s=s, Y=Y, F=F, seed=seed)
    if kind == "solve":
        p, ref, x, q, fe, V, F = _solve_inputs(case, seed)
        s = _context(p, ref, x, q, fe, stream, False)
        s.fill_all_blob_pos()
        s.set_up_gaussians()
        s.calculate_forces()
        rhs = np.concatenate([-V, -s.multiply_by_KT_at_midstep(F) - fe])
        return dict(case=case, s=s, rhs=torch.from_numpy(rhs).cuda())
    if kind == "step":
        p, ref, x, q, fe = _placed(case["channel"], case["bodies"], case["blobs"], case["grid"], case["box"])
        return dict(_stepped(p, ref, x, q, fe, case, seed, stream), case=case)
    members = [_stepped(*_member(case["first"] + i), case, seed + 1000 * i, torch.cuda.Stream())
               for i in range(case["members"])]
    return dict(case=case, members=members, seeds=[m["seed"] for m in members])


# ------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "mobility":
        s, n = state["s"], state["F"].numel()
        V = torch.empty(n, dtype=torch.float64, device="cuda")
        if case["fresh"]:
            s.set_up_gaussians(state["Y"])
        if case["precision"] == 0:
            return s.apply_mobility(state["F"], out=V)
        s.spread(state["F"], 1)
        s.stokes_solve(1)
        return s.interp(1, out=V).float()
    if kind == "noise":
        s = state["s"]
        V = torch.empty(state["F"].numel(), dtype=torch.float64, device="cuda")
        s.produce_random_velocity_field(state["seed"], 3)
        return s.calculate_random_blob_velocities(out=V)
    if kind == "solve":
        s = state["s"]
        soln = torch.empty(state["rhs"].numel(), dtype=torch.float64, device="cuda")
        s.set_RHS(state["rhs"])
        return s.invert_saddle_point_system(out=soln)[1]
    if kind == "step":
        s = state["s"]
        s.set_bodies(state["x"], state["q"])
        s.step_async(state["seed"], 1)
        s.step_wait()
        return s.get_bodies()
    for m in state["members"]:
        m["s"].set_bodies(m["x"], m["q"])
    step_many([m["s"] for m in state["members"]], state["seeds"], 1)
    return [m["s"].get_bodies() for m in state["members"]]


# ------------------------------------------------------------------ what a pass cannot do without
def _product(nb, nx, ny, nz, size):
    """Bytes and operations of one mobility product.  Whatever the order of the passes, a three-dimensional transform
    of a grid larger than the cache writes and reads its half spectrum once before the last direction and once after
    it; the forces, positions and velocities of the blobs come on top.  Operations: the separable stencils (W^3
    points, 3 components, multiply and add, twice), the transforms (5/2 n log2 n, both ways), the projection."""
    G = nx * ny * nz
    Gc = nx * ny * (nz // 2 + 1)
    data = 4 * 3 * Gc * 2 * size + 3 * 3 * nb * 8
    flops = 2 * nb * 20 ** 3 * 3 * 2 + 2 * 3 * 2.5 * G * math.log2(G) + 30 * Gc
    return data, flops


def work(case):
    kind = case["kind"]
    size = 4 if case["precision"] == 1 else 8
    if kind in ("mobility", "noise"):
        nb = case["bodies"] * case["blobs"]
        data, flops = _product(nb, case["nx"], case["ny"], case["nz"], size)
        if kind == "noise":  # no spread and no forward transform
            data, flops = data / 2, flops / 2
        return {"bytes": data, "flops": flops}
    if kind in ("solve", "step"):
        nb, g, rounds = case["bodies"] * case["blobs"], case["grid"], 20
        if kind == "step" and case["algorithm"] == 1:
            rounds += 12
        data, flops = _product(nb, g, g, g, size)
        return {"bytes": rounds * data, "flops": rounds * flops}
    total = {"bytes": 0.0, "flops": 0.0}
    for i in range(case["members"]):
        M, phi = _member_size(case["first"] + i)
        g = configs.nearest_fft_size(1.86 * configs.box_for_volume_fraction(6 * M, phi))
        data, flops = _product(6 * M, g, g, g, size)
        total["bytes"] += 20 * data
        total["flops"] += 20 * flops
    return total


def _member_size(i):
    rng = np.random.default_rng(i)
    return int(rng.integers(50, 501)), float(rng.uniform(0.05, 0.20))


# ------------------------------------------------------------------ the result in 64 bits
class _Plain:
    """The mobility in plain torch, FP64: Gaussians of W points per dimension, transforms of the half spectrum whose
    inverse along z drops the imaginary parts of its first and last plane (even sides)."""

    def __init__(self, n, dx, Y, W=20, a=1.0, eta=1.0):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.n, self.dx, self.W, self.eta = n, dx, W, eta
        Y = torch.as_tensor(Y, dtype=torch.float64, device=self.dev).reshape(-1, 3)
        N = torch.tensor(n, device=self.dev)
        g = (Y / dx).to(torch.int64)[:, :, None] - W // 2 + 1 + torch.arange(W, device=self.dev)
        self.w = torch.exp(-math.pi * (g.to(torch.float64) * dx - Y[:, :, None]) ** 2 / (2 * a * a)) / (math.sqrt(2.0) * a)
        self.i = g % N[None, :, None]

    def _chunks(self):
        B = 2048
        for b in range(0, len(self.w), B):
            w, i = self.w[b:b + B], self.i[b:b + B]
            ker = w[:, 0, :, None, None] * w[:, 1, None, :, None] * w[:, 2, None, None, :]
            at = (i[:, 0, :, None, None] * self.n[1] + i[:, 1, None, :, None]) * self.n[2] + i[:, 2, None, None, :]
            yield b, min(len(self.w), b + B), ker.reshape(len(w), -1), at.reshape(len(w), -1)

    def spread(self, F):
        F = torch.as_tensor(F, dtype=torch.float64, device=self.dev).reshape(-1, 3)
        grid = torch.zeros(3, self.n[0] * self.n[1] * self.n[2], dtype=torch.float64, device=self.dev)
        for b, e, ker, at in self._chunks():
            for c in range(3):
                grid[c].index_add_(0, at.reshape(-1), (ker * F[b:e, c:c + 1]).reshape(-1))
        return grid.reshape(3, *self.n)

    def solve(self, grid):
        q, nz = [], self.n[2]
        for d, n in enumerate(self.n):
            k = torch.arange(n if d < 2 else nz // 2 + 1, device=self.dev)
            k = torch.where(k <= n // 2, k, k - n).to(torch.float64) * (2.0 * math.pi / (self.dx * n))
            q.append(k.reshape([-1 if e == d else 1 for e in range(3)]))
        inv = 1.0 / (q[0] ** 2 + q[1] ** 2 + q[2] ** 2 + 1e-16)
        inv[0, 0, 0] = 0.0
        f = [torch.fft.rfftn(grid[c]) for c in range(3)]
        kf = (q[0] * f[0] + q[1] * f[1] + q[2] * f[2]) * inv
        for c in range(3):
            u = torch.fft.ifft2((f[c] - q[c] * kf) * inv / self.eta, dim=(0, 1))
            u[:, :, 0].imag = 0.0
            u[:, :, nz // 2].imag = 0.0
            grid[c] = torch.fft.irfft(u, n=nz, dim=2)
        return grid

    def interp(self, grid):
        V = torch.zeros(len(self.w), 3, dtype=torch.float64, device=self.dev)
        flat = grid.reshape(3, -1)
        for b, e, ker, at in self._chunks():
            for c in range(3):
                V[b:e, c] = (flat[c][at] * ker).sum(1)
        return V.reshape(-1) * self.dx ** 3

    def apply(self, F):
        return self.interp(self.solve(self.spread(F)))


def exact(case, seed):
    kind = case["kind"]
    if kind == "mobility":
        _, Y, F = _cloud(case, seed)
        if not torch.cuda.is_available() and case["nx"] * case["ny"] * case["nz"] > 128 ** 3:
            return None
        return _Plain((case["nx"], case["ny"], case["nz"]), case["dx"], Y).apply(F)
    if kind != "solve" or case["bodies"] * case["blobs"] > 200 and not torch.cuda.is_available():
        return None  # noise drawn by the library, or steps with it
    p, ref, x, q, fe, V, F = _solve_inputs(case, seed)
    r = torch.einsum("nij,mj->nmi", _rotations(q.reshape(-1, 4)), torch.from_numpy(np.asarray(ref)).reshape(-1, 3))
    Y = (torch.from_numpy(x).reshape(-1, 1, 3) + r).reshape(-1, 3)
    L = torch.tensor(p.box, dtype=torch.float64)
    Y = Y - L * torch.floor(Y / L)
    plain = _Plain((p.nx, p.ny, p.nz), p.dx, Y)
    n3, n6 = 3 * p.num_blobs, 6 * p.num_bodies
    A = torch.zeros(n3 + n6, n3 + n6, dtype=torch.float64)
    unit = torch.zeros(n3, dtype=torch.float64)
    for k in range(n3):
        unit[k] = 1.0
        A[:n3, k] = plain.apply(unit).cpu()
        unit[k] = 0.0
    K = torch.zeros(n3, n6, dtype=torch.float64)
    for b in range(p.num_blobs):
        n, (rx, ry, rz) = b // p.blobs_per_body, r.reshape(-1, 3)[b].tolist()
        K[3 * b:3 * b + 3, 6 * n:6 * n + 3] = torch.eye(3, dtype=torch.float64)
        K[3 * b:3 * b + 3, 6 * n + 3:6 * n + 6] = torch.tensor([[0, rz, -ry], [-rz, 0, rx], [ry, -rx, 0]])
    A[:n3, n3:], A[n3:, :n3] = -K, -K.T
    rhs = torch.cat([torch.from_numpy(-V), -K.T @ torch.from_numpy(F) - torch.from_numpy(fe)])
    # straight rods leave the spin about their axis free: the solution without it
    return torch.linalg.lstsq(A, rhs[:, None], rcond=1e-10, driver="gelsd").solution[:, 0]
