"""The work that users of this framework have it do, as measurable cases.

A case is one of five kinds of call, each over the range of sizes that the
tests, the benchmark configurations and the reference's own projects cover:

  md        one System: advance some steps (NVE, Nose-Hoover or Langevin; FP64
            or FP32-mixed), read the energies and the frame, as a project's
            main loop does between two observations
  slab      the same on a liquid slab in its vapour (uneven cell occupancy)
  ensemble  one Ensemble of replicas of different size, density and temperature
  point     a single-point evaluation: new positions in, list, forces,
            energies and pair counts out
  adjoint   a trajectory loss and its gradients

Frames go to page-locked host buffers, as a program that reads many of them
keeps them.  All inputs come from the seed alone and are made on the GPU.
"""
import ctypes
import math

import numpy as np
import torch

import mdacp_b200 as M
from mdacp_b200 import adjoint

PRECISION = {"fp64": M.FP64, "mixed": M.FP32_MIXED}
THERMOSTAT = {"nve": M.NVE, "nose_hoover": M.NOSE_HOOVER, "langevin": M.LANGEVIN}
TAU, GAMMA = 0.1, 1.0
SKIN = 0.3


# ------------------------------------------------------------------ the cases
def _md(nx, ny, nz, vacancies, rho, temp, rc, dt, precision, thermostat, steps, **name):
    return dict(kind="md", nx=nx, ny=ny, nz=nz, vacancies=vacancies, rho=rho, temp=temp, rc=rc, dt=dt,
                precision=precision, thermostat=thermostat, steps=steps, **name)


def listed():
    return [
        # the smallest call: a program that couples to the system and takes it one step at a time
        _md(6, 6, 6, 0, 0.8, 1.0, 2.5, 0.005, "fp64", "nve", 1, name="md_864_fp64_step"),
        # the plain 32,000-atom benchmark system, between two observations
        _md(20, 20, 20, 0, 0.5, 1.0, 2.5, 0.005, "mixed", "nve", 100, name="md_32000_mixed"),
        # thermalisation of a mid-size liquid, odd in every way
        _md(31, 29, 33, 7, 0.7, 0.9, 2.5, 0.005, "fp64", "nose_hoover", 60, name="md_118661_fp64_nosehoover"),
        # a mid-size production run
        _md(41, 39, 40, 13, 0.8442, 0.722, 2.5, 0.004, "mixed", "nve", 100, name="md_255827_mixed"),
        # the large homogeneous liquid, in both precisions
        _md(80, 80, 80, 0, 0.8442, 0.722, 2.5, 0.004, "mixed", "nve", 100, name="md_2048000_mixed"),
        _md(80, 80, 80, 0, 0.8442, 0.722, 2.5, 0.004, "fp64", "nve", 50, name="md_2048000_fp64"),
        # liquid-vapour coexistence under Langevin noise
        dict(kind="slab", nx=61, rho=0.75, rho_vapour=0.02, temp=0.9, rc=3.0, dt=0.005, precision="mixed",
             thermostat="langevin", steps=60, name="slab_980k_langevin"),
        # a scan of state points, one launch for all replicas
        dict(kind="ensemble", replicas=256, n_low=500, n_high=20000, rho_low=0.3, rho_high=0.9, temp_low=0.7,
             temp_high=1.5, rc=2.5, dt=0.005, precision="mixed", steps=100, name="ensemble_256_mixed"),
        # a small scan in FP64, boxes down to all-pairs size
        dict(kind="ensemble", replicas=24, n_low=500, n_high=3000, rho_low=0.3, rho_high=0.9, temp_low=0.7,
             temp_high=1.5, rc=2.5, dt=0.005, precision="fp64", steps=100, name="ensemble_24_fp64"),
        # energies and forces of given configurations
        dict(kind="point", nx=40, ny=40, nz=40, vacancies=0, rho=0.8442, temp=0.722, rc=2.5, dt=0.005,
             precision="fp64", name="point_256000_fp64"),
        # differentiable trajectories: the full-size fit, and a small one in an optimiser's loop
        dict(kind="adjoint", nx=20, ny=20, nz=20, rho=0.8442, temp=1.0, rc=2.5, dt=0.005, steps=200, every=20,
             gradients=True, name="adjoint_32000"),
        dict(kind="adjoint", nx=5, ny=5, nz=5, rho=0.8442, temp=1.0, rc=2.5, dt=0.005, steps=50, every=10,
             gradients=True, name="adjoint_500"),
    ]


def _edges(n, least, rng):
    """Three lattice edges, not all equal, whose block holds about n atoms."""
    e = (n / 4.0) ** (1.0 / 3.0)
    edges = [max(least, round(e * rng.uniform(0.85, 1.15))) for _ in range(2)]
    return edges + [max(least, round(n / (4.0 * edges[0] * edges[1])))]


def _least_edge(rho, reach, cells=3):
    """Lattice cells along an axis that hold `cells` cells of `reach`."""
    return math.ceil(cells * reach / (4.0 / rho) ** (1.0 / 3.0) + 1e-9)


def draw(rng):
    kind = rng.choice(["md", "md", "md", "slab", "ensemble", "point", "adjoint"])
    rho, temp, dt = round(rng.uniform(0.3, 0.9), 3), round(rng.uniform(0.7, 1.5), 3), rng.choice([0.004, 0.005])
    rc, precision = rng.choice([2.5, 2.5, 3.0]), rng.choice(["fp64", "mixed"])

    def size(low, high):
        return math.exp(rng.uniform(math.log(low), math.log(high)))

    if kind in ("md", "point"):
        nx, ny, nz = _edges(size(800, 1.5e6), _least_edge(rho, rc + SKIN), rng)
        box = dict(nx=nx, ny=ny, nz=nz, vacancies=rng.randrange(0, 32), rho=rho, temp=temp, rc=rc, dt=dt,
                   precision=precision)
        if kind == "point":
            return dict(kind=kind, **box)
        atoms = 4 * nx * ny * nz
        steps = rng.choice([1, 7, 20, 50, 100])
        steps = max(1, min(steps, int((5e7 if precision == "fp64" else 1e8) / atoms)))
        return dict(kind=kind, thermostat=rng.choice(["nve", "nve", "nose_hoover", "langevin"]), steps=steps, **box)
    if kind == "slab":
        return dict(kind=kind, nx=int(size(14, 60)), rho=round(rng.uniform(0.65, 0.8), 3), rho_vapour=0.02,
                    temp=0.9, rc=3.0, dt=0.005, precision=precision, thermostat=rng.choice(["nve", "langevin"]),
                    steps=rng.choice([5, 20, 40]))
    if kind == "ensemble":
        high = int(size(1500, 20000))
        replicas = max(2, int(size(2, min(256, 2.2e6 / high))))
        return dict(kind=kind, replicas=replicas, n_low=500, n_high=high, rho_low=0.3, rho_high=0.9, temp_low=0.7,
                    temp_high=1.5, rc=2.5, dt=0.005, precision=precision, steps=rng.choice([1, 20, 50, 100]))
    rho, steps = round(rng.uniform(0.5, 0.9), 3), int(size(5, 150))
    nx, ny, nz = _edges(size(500, 30000), _least_edge(rho, 2.5), rng)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, rho=rho, temp=temp, rc=2.5, dt=0.005, steps=steps,
                every=max(1, min(steps, rng.choice([5, 10, 20]))), gradients=rng.random() < 0.75)


# ----------------------------------------------------------------- the inputs
def _generator(seed):
    return torch.Generator("cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _lattice(nx, ny, nz, a, basis):
    z, y, x = torch.meshgrid(*(torch.arange(k, device="cuda", dtype=torch.float64) for k in (nz, ny, nx)),
                             indexing="ij")
    cells = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], dim=1)
    b = torch.tensor(basis, device="cuda", dtype=torch.float64)
    return ((cells[:, None, :] + b[None] + 0.25) * a).reshape(-1, 3)


FCC = [[0.0, 0.0, 0.0], [0.0, 0.5, 0.5], [0.5, 0.0, 0.5], [0.5, 0.5, 0.0]]


def _jittered(q, a, L, jitter, g):
    """Lattice sites moved by up to jitter lattice constants per axis, inside the box."""
    q = q + (torch.rand(q.shape, generator=g, device="cuda", dtype=torch.float64) * 2.0 - 1.0) * (jitter * a)
    q = torch.remainder(q, L)
    return torch.where(q >= L, torch.zeros_like(q), q)


def _velocities(n, temp, g):
    v = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    v -= v.mean(dim=0)
    return v * math.sqrt(3.0 * n * temp / float((v * v).sum()))


def _liquid(nx, ny, nz, vacancies, rho, temp, g):
    """Positions, velocities and box of a jittered lattice with some sites left out."""
    a = (4.0 / rho) ** (1.0 / 3.0)
    L = torch.tensor([nx * a, ny * a, nz * a], device="cuda", dtype=torch.float64)
    q = _jittered(_lattice(nx, ny, nz, a, FCC), a, L, 0.05, g)
    if vacancies:
        keep = torch.ones(q.shape[0], dtype=torch.bool, device="cuda")
        keep[torch.randperm(q.shape[0], generator=g, device="cuda")[:vacancies]] = False
        q = q[keep]
    return q, _velocities(q.shape[0], temp, g), L


def _slab(case, g):
    """A liquid cube in the middle quarter of a 1:1:4 box, vapour in the rest."""
    nx, a = case["nx"], (4.0 / case["rho"]) ** (1.0 / 3.0)
    edge = nx * a
    L = torch.tensor([edge, edge, 4.0 * edge], device="cuda", dtype=torch.float64)
    up = torch.tensor([0.0, 0.0, 1.5 * edge], device="cuda", dtype=torch.float64)
    liquid = _jittered(_lattice(nx, nx, nx, a, FCC) + up, a, L, 0.05, g)
    m = max(1, int(edge * case["rho_vapour"] ** (1.0 / 3.0)))
    s = edge / m  # vapour sites, at least a diameter away from the liquid's faces
    vapour = _lattice(m, m, 4 * m, s, [[0.25, 0.25, 0.25]])
    vapour = vapour[(vapour[:, 2] < 1.5 * edge - 0.5 * s) | (vapour[:, 2] > 2.5 * edge + 0.5 * s)]
    q = torch.cat([liquid, _jittered(vapour, s, L, 0.2, g)])
    return q, _velocities(q.shape[0], case["temp"], g), L


def _replicas(case, g):
    """(q, v, L) of every replica; sizes and state points spread evenly over the case's ranges (a Kronecker
    sequence, so that every seed has the same), positions and velocities from the seed."""
    out = []
    for k in range(case["replicas"]):
        a, b, c = ((0.5 + k * x) % 1.0 for x in (0.8191725134, 0.6710436067, 0.5497004779))
        n = case["n_low"] + a * (case["n_high"] - case["n_low"])
        rho = case["rho_low"] + b * (case["rho_high"] - case["rho_low"])
        temp = case["temp_low"] + c * (case["temp_high"] - case["temp_low"])
        nx = max(round((n / 4.0) ** (1.0 / 3.0)), _least_edge(rho, case["rc"] + SKIN, 2))
        nz = max(round(n / (4.0 * nx * nx)), _least_edge(rho, case["rc"] + SKIN, 2))
        out.append(_liquid(nx, nx, nz, 0, rho, temp, g))
    return out


def _inputs(case, seed):
    g = _generator(seed)
    if case["kind"] == "slab":
        return _slab(case, g)
    if case["kind"] == "ensemble":
        return _replicas(case, g)
    return _liquid(case["nx"], case["ny"], case["nz"], case.get("vacancies", 0), case["rho"], case["temp"], g)


def _pinned(*shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _pinned_frame(x):
    out = _pinned(x.shape[0], 4)
    out[:, :3] = x.cpu().numpy()
    out[:, 3] = 0.0
    return out


def prepare(case, seed):
    x = _inputs(case, seed)
    state = {"case": case}
    if case["kind"] == "ensemble":
        states = [(q.cpu().numpy(), v.cpu().numpy(), L.cpu().numpy()) for q, v, L in x]
        ens = M.Ensemble(states, cutoff=case["rc"], time_step=case["dt"], precision=PRECISION[case["precision"]])
        n = ens.ntot
        return dict(state, ens=ens, q4=_pinned(n, 4), v4=_pinned(n, 4), ids=_pinned(n, dtype=torch.int32))
    q, v, L = x
    n = q.shape[0]
    if case["kind"] == "adjoint":
        return dict(state, q=q.cpu().numpy(), v=v.cpu().numpy(), L=L.cpu().numpy())
    system = M.System(L.tolist(), cutoff=case["rc"], time_step=case["dt"], capacity=n,
                      precision=PRECISION[case["precision"]],
                      thermostat=THERMOSTAT[case.get("thermostat", "nve")], aimed_temperature=case["temp"],
                      heatbath_tau=TAU, heatbath_gamma=GAMMA, seed=int(seed))
    state.update(system=system, q4=_pinned_frame(q), v4=_pinned_frame(v))
    if case["kind"] == "point":
        return dict(state, f4=_pinned(n, 4))
    system.set_state4(state["q4"], state["v4"])
    return state


# ------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    if case["kind"] == "adjoint":
        options = dict(steps=case["steps"], checkpoint_every=case["every"], time_step=case["dt"], cutoff=case["rc"])
        if not case["gradients"]:
            return {"loss": adjoint.trajectory_loss(state["q"], state["v"], state["L"], **options)}
        loss, de, ds, dq = adjoint.trajectory_gradients(state["q"], state["v"], state["L"], **options)
        return {"loss": loss, "d_epsilon": de, "d_sigma": ds, "d_q": dq}
    if case["kind"] == "ensemble":
        ens = state["ens"]
        ens.calculate(case["steps"])
        ke, pe, virial = ens.observe()
        # the C ABI's readout into the program's own buffers
        dp, ip = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int)
        st = ens.lib.mdg_ensemble_get_state(ens.h, state["q4"].ctypes.data_as(dp), state["v4"].ctypes.data_as(dp),
                                            state["ids"].ctypes.data_as(ip))
        if st != 0:
            raise M.MdgError(st, "mdg_ensemble_get_state")
        return {"ke": ke, "pe": pe, "virial": virial, "q": state["q4"], "v": state["v4"], "ids": state["ids"]}
    system = state["system"]
    if case["kind"] == "point":
        system.set_state4(state["q4"], state["v4"])
        system.make_pairlist()
        st = system.lib.mdg_forces(system.h, state["f4"].ctypes.data_as(ctypes.POINTER(ctypes.c_double)))
        if st != 0:
            raise M.MdgError(st, "mdg_forces")
        ke, pe, virial = system.observe()
        within, entries = system.pair_counts()
        return {"ke": ke, "pe": pe, "virial": virial, "f": state["f4"], "ids": system.ids(), "within": within,
                "entries": entries}
    system.calculate(case["steps"])
    ke, pe, virial = system.observe()
    system.get_state4(state["q4"], state["v4"])
    return {"ke": ke, "pe": pe, "virial": virial, "q": state["q4"], "v": state["v4"], "ids": system.ids()}


def _atoms(case):
    """Atoms and mean density (of the pairs) of a case."""
    if case["kind"] == "ensemble":
        return (0.5 * (case["n_low"] + case["n_high"]) * case["replicas"],
                0.5 * (case["rho_low"] + case["rho_high"]))
    n = 4.0 * case["nx"] * case.get("ny", case["nx"]) * case.get("nz", case["nx"])
    return n - case.get("vacancies", 0), case["rho"]


def work(case):
    """Bytes: every step reads and writes positions and velocities (96 B an atom); an evaluation reads positions
    and writes forces.  Flops: about 30 for each pair within the cut-off, counted once; twice that for the loss
    and its gradient, three times for a Hessian-vector product."""
    n, rho = _atoms(case)
    pairs = 0.5 * n * rho * 4.0 / 3.0 * math.pi * case["rc"] ** 3
    if case["kind"] == "point":
        return {"bytes": 96.0 * n, "flops": 60.0 * pairs}
    if case["kind"] == "adjoint":
        each = 30.0 * (1 + 2) if not case["gradients"] else 30.0 * (1 + 2 + 1 + 2 + 3)
        sweeps = 3 if case["gradients"] else 1  # forward, recomputed segment, reverse
        return {"bytes": 96.0 * n * case["steps"] * sweeps, "flops": each * pairs * case["steps"]}
    return {"bytes": 96.0 * n * case["steps"], "flops": 30.0 * pairs * case["steps"]}


# ------------------------------------------------- the same in plain 64 bits
def _near(q, L, reach):
    """Pairs (i, j), each once, closer than `reach` in the periodic box (minimum image)."""
    n, dev = q.shape[0], q.device
    ms = [int(x / reach) for x in L.tolist()]
    if min(ms) < 3:
        i, j = torch.triu_indices(n, n, 1, device=dev)
        d = q[i] - q[j]
        d -= L * torch.round(d / L)
        keep = (d * d).sum(1) < reach * reach
        return i[keep], j[keep]
    m = torch.tensor(ms, device=dev)
    c = torch.minimum((torch.remainder(q, L) / L * m).long(), m - 1)
    cell = (c[:, 2] * ms[1] + c[:, 1]) * ms[0] + c[:, 0]
    order = torch.argsort(cell)
    count = torch.bincount(cell, minlength=ms[0] * ms[1] * ms[2])
    start = torch.cumsum(count, 0) - count
    width = int(count.max())
    slots = torch.arange(width, device=dev)
    table = torch.full((count.numel(), width), -1, dtype=torch.long, device=dev)
    rank = torch.arange(n, device=dev) - start[cell[order]]
    table[cell[order], rank] = order
    z, y, x = torch.meshgrid(*(torch.arange(k, device=dev) for k in (ms[2], ms[1], ms[0])), indexing="ij")
    x, y, z = x.reshape(-1), y.reshape(-1), z.reshape(-1)
    half = [(0, 0, 0)] + [(dx, dy, dz) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)
                          if (dz, dy, dx) > (0, 0, 0)]
    got_i, got_j = [], []
    chunk = max(1, 40_000_000 // (width * width))
    for dx, dy, dz in half:
        other = ((z + dz) % ms[2] * ms[1] + (y + dy) % ms[1]) * ms[0] + (x + dx) % ms[0]
        for a in range(0, count.numel(), chunk):
            ti, tj = table[a:a + chunk, :, None], table[other[a:a + chunk]][:, None, :]
            keep = (ti >= 0) & (tj >= 0)
            if (dx, dy, dz) == (0, 0, 0):
                keep &= slots[:, None] < slots[None, :]
            ti, tj = ti.expand(keep.shape)[keep], tj.expand(keep.shape)[keep]
            d = q[ti] - q[tj]
            d -= L * torch.round(d / L)
            keep = (d * d).sum(1) < reach * reach
            got_i.append(ti[keep])
            got_j.append(tj[keep])
    return torch.cat(got_i), torch.cat(got_j)


class _Plain:
    """One or several periodic systems in FP64: pairs listed a skin wide, listed anew when an atom has moved half of it."""

    def __init__(self, systems, rc):
        self.systems = systems  # (first atom, end, L)
        self.rc, self.skin = rc, 0.5
        self.Lp = None
        s6 = rc ** -6
        self.c2 = 6.0 * s6 * s6 / rc ** 2 - 3.0 * s6 / rc ** 2
        self.c0 = -s6 * s6 + s6 - self.c2 * rc * rc

    def pairs(self, q):
        """Pairs (i, j) and their displacement, of those within the cut-off."""
        if self.Lp is not None:
            moved = float(((q - self.q0) ** 2).sum(1).max())
        if self.Lp is None or moved > 0.25 * self.skin ** 2:
            found = [(a, L) + _near(q[a:b], L, self.rc + self.skin) for a, b, L in self.systems]
            self.i = torch.cat([a + i for a, _, i, _ in found])
            self.j = torch.cat([a + j for a, _, _, j in found])
            self.Lp = found[0][1] if len(found) == 1 else torch.cat([L.expand(i.numel(), 3) for _, L, i, _ in found])
            self.q0 = q.clone()
        d = q[self.i] - q[self.j]
        d -= self.Lp * torch.round(d / self.Lp)
        near = (d * d).sum(1) <= self.rc * self.rc
        return self.i[near], self.j[near], d[near]

    def forces(self, q):
        i, j, d = self.pairs(q)
        r2 = (d * d).sum(1)
        r6 = r2 ** 3
        f = ((48.0 - 24.0 * r6) / (r6 * r6 * r2) - 8.0 * self.c2)[:, None] * d
        return torch.zeros_like(q).index_add_(0, i, f).index_add_(0, j, -f)

    def sums(self, q, v):
        """Kinetic energy, potential energy and virial (a third of sum df r^2) per system."""
        i, _, d = self.pairs(q)
        r2 = (d * d).sum(1)
        r6 = r2 ** 3
        e = 4.0 * (1.0 / (r6 * r6) - 1.0 / r6 + self.c2 * r2 + self.c0)
        w = ((24.0 * r6 - 48.0) / (r6 * r6 * r2) + 8.0 * self.c2) * r2
        per = [0.5 * (v * v).sum(1), torch.zeros_like(v[:, 0]).index_add_(0, i, e),
               torch.zeros_like(v[:, 0]).index_add_(0, i, w)]
        ke, pe, vir = (torch.stack([x[a:b].sum() for a, b, _ in self.systems]) for x in per)
        return ke, pe, vir / 3.0


def _normals(seed, n, step):
    """Three standard normals per atom: Philox4x32-10 at (id, step), key = seed, then Box-Muller."""
    m = 0xFFFFFFFF
    c = [torch.arange(n, device="cuda"), torch.full((n,), step & m, device="cuda"),
         torch.full((n,), step >> 32, device="cuda"), torch.full((n,), 0x4C414E47, device="cuda")]
    k0, k1 = seed & m, (seed >> 32) & m

    def mul(a, x):  # 32 x 32 -> (high, low) words, in 16-bit parts
        lo, hi = a * (x & 0xFFFF), a * (x >> 16)
        low = lo + ((hi & 0xFFFF) << 16)
        return ((hi >> 16) + (low >> 32)) & m, low & m

    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    u = [(x.double() + 0.5) * 2.0 ** -32 for x in c]
    r0, r1 = torch.sqrt(-2.0 * torch.log(u[0])), torch.sqrt(-2.0 * torch.log(u[2]))
    return torch.stack([r0 * torch.cos(2.0 * math.pi * u[1]), r0 * torch.sin(2.0 * math.pi * u[1]),
                        r1 * torch.cos(2.0 * math.pi * u[3])], dim=1)


def _advance(plain, q, v, case, seed):
    dt, n, zeta, temp = case["dt"], q.shape[0], 0.0, case.get("temp")
    kind = case.get("thermostat", "nve")
    for t in range(case["steps"]):
        q = q + v * (dt / 2)
        if kind == "nose_hoover":
            zeta += (float((v * v).sum()) / (3.0 * n) - temp) / TAU ** 2 * (dt / 2)
            s = math.exp(-dt / 2 * zeta)
            v = (v * s + plain.forces(q) * dt) * s
            zeta += (float((v * v).sum()) / (3.0 * n) - temp) / TAU ** 2 * (dt / 2)
        else:
            v = v + plain.forces(q) * dt
        if kind == "langevin":
            v = v + (-GAMMA * v + math.sqrt(2.0 * GAMMA * temp / dt) * _normals(int(seed), n, t)) * dt
        else:
            q = q + v * (dt / 2)
    return q, v


def _loss(plain, q, n, steps):
    """The trajectory loss's term of one state: potential energy and smoothed pair count of the shell 1.0 < r < 1.5."""
    def term(q, eps, sigma):
        i, j, _ = plain.pairs(q.detach())
        d = q[i] - q[j]
        d = d - plain.systems[0][2] * torch.round(d.detach() / plain.systems[0][2])
        r2 = (d * d).sum(1)
        s2 = r2 / sigma ** 2
        s6 = s2 ** -3
        r = torch.sqrt(r2)
        near = torch.sigmoid((r - 1.0) / 0.05) * torch.sigmoid((1.5 - r) / 0.05)
        return ((4.0 * eps * (s6 * s6 - s6 + plain.c2 * s2 + plain.c0)).sum() + near.sum()) / (steps * n)
    return term


def _force_of(plain, q, eps, sigma):
    i, j, _ = plain.pairs(q.detach())
    d = q[i] - q[j]
    d = d - plain.systems[0][2] * torch.round(d.detach() / plain.systems[0][2])
    s2 = (d * d).sum(1) / sigma ** 2
    s6 = s2 ** 3
    f = (eps / sigma ** 2 * ((48.0 - 24.0 * s6) / (s6 * s6 * s2) - 8.0 * plain.c2))[:, None] * d
    return torch.zeros_like(q).index_add(0, i, f).index_add(0, j, -f)


def _exact_adjoint(case, q, v, L):
    n, T, dt = q.shape[0], case["steps"], case["dt"]
    plain = _Plain([(0, n, L)], case["rc"])
    eps, sigma = (torch.tensor(1.0, dtype=torch.float64, device="cuda", requires_grad=True) for _ in range(2))
    term = _loss(plain, q, n, T)
    kept, loss = [], 0.0
    with torch.no_grad():
        for _ in range(T):
            kept.append((q, v))
            qh = q + v * (dt / 2)
            v = v + _force_of(plain, qh, eps, sigma) * dt
            q = qh + v * (dt / 2)
            loss += float(term(q, eps, sigma))
    if not case["gradients"]:
        return {"loss": loss}
    lq, lv, de, ds = torch.zeros_like(q), torch.zeros_like(v), 0.0, 0.0
    for q, v in reversed(kept):
        q, v = q.requires_grad_(True), v.requires_grad_(True)
        qh = q + v * (dt / 2)
        v1 = v + _force_of(plain, qh, eps, sigma) * dt
        q1 = qh + v1 * (dt / 2)
        g = torch.autograd.grad((q1 * lq).sum() + (v1 * lv).sum() + term(q1, eps, sigma), (q, v, eps, sigma))
        lq, lv, de, ds = g[0], g[1], de + float(g[2]), ds + float(g[3])
    return {"loss": loss, "d_epsilon": de, "d_sigma": ds, "d_q": lq.cpu().numpy()}


def exact(case, seed):
    x = _inputs(case, seed)
    if case["kind"] == "ensemble":
        ends = np.cumsum([q.shape[0] for q, _, _ in x]).tolist()
        if ends[-1] * case["steps"] > 3e7:
            return None  # too long
        plain = _Plain([(b - q.shape[0], b, L) for (q, _, L), b in zip(x, ends)], case["rc"])
        q, v = _advance(plain, torch.cat([q for q, _, _ in x]), torch.cat([v for _, v, _ in x]), case, seed)
        ke, pe, vir = plain.sums(q, v)
        return {"ke": ke.cpu().numpy(), "pe": pe.cpu().numpy(), "virial": vir.cpu().numpy(), "q": None, "v": None,
                "ids": None}
    q, v, L = x
    n = q.shape[0]
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, q, v, L)
    plain = _Plain([(0, n, L)], case["rc"])
    if case["kind"] == "point":
        ke, pe, vir = (float(s) for s in plain.sums(q, v))
        # forces in slot order: by cell (z, y, x), then x, then upload index
        ms = [int(s / (case["rc"] + SKIN)) for s in L.tolist()]
        h = q.cpu().numpy()
        c = np.stack([np.minimum((h[:, d] * (ms[d] / float(L[d]))).astype(np.int64), ms[d] - 1) for d in range(3)])
        order = np.lexsort((np.arange(n), h[:, 0], (c[2] * ms[1] + c[1]) * ms[0] + c[0]))
        f = np.zeros((n, 4))
        f[:, :3] = plain.forces(q).cpu().numpy()[order]
        within = 2 * plain.pairs(q)[0].numel()
        return {"ke": ke, "pe": pe, "virial": vir, "f": f, "ids": None, "within": within, "entries": None}
    if n * case["steps"] > 6e7:
        return None  # too long
    q, v = _advance(plain, q, v, case, seed)
    ke, pe, vir = (float(s) for s in plain.sums(q, v))
    return {"ke": ke, "pe": pe, "virial": vir, "q": None, "v": None, "ids": None}
