"""What the performance of this repository is measured on: passes of the time step as its users run them.

A pass is what a program does between two outputs: some cycles of the Lagrange + remap step on a state in the middle of
a run, through the public entry points, then the fields read back into the program's pinned host buffers.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "arcane-benchs_b200"))

import mhy_b200  # noqa: E402
from mhy_b200 import Batch, Context, gen  # noqa: E402

LIMITERS = {"minmod": 0, "superBee": 1, "vanLeer": 2, "minmodG": 3, "superBeeG": 4, "vanLeerG": 5}
FIELDS = ("density", "internal_energy", "pressure", "velocity")


def _case(problem, nx, ny, nz, cycles, lead, **options):
    """lead: cycles run before the pass, so that it meets a developed flow and not the state at rest of t = 0."""
    c = {"problem": problem, "nx": nx, "ny": ny, "nz": nz, "cycles": cycles, "lead": lead, "drive": "step",
         "precision": "fp64", "order": 2, "limiter": "minmod", "csts": False, "pente_borne": False,
         "total_energy": False, "fractions": False, "instances": 1}
    c.update(options)
    return c


def listed():
    return [
        # A host code that owns its device fields and asks for the CFL time step alone: the smallest call there is.
        dict(_case("dt", 100, 5, 5, 1, 0), name="dt of device fields 100x5x5"),
        # The same call on the mesh of the headline run.
        dict(_case("dt", 128, 128, 128, 1, 0), name="dt of device fields 128^3"),
        # The shock tube of the reference's decks, driven entry point by entry point from the host as the module's
        # time loop drives it, dt read every cycle: launches and host reads are what counts.
        dict(_case("sod", 100, 5, 5, 20, 30, drive="entry points"), name="Sod 100x5x5 coupled"),
        # A small 3D run of the kind that parameter studies are made of.
        dict(_case("sedov", 37, 37, 37, 20, 40, limiter="superBee"), name="Sedov 37^3"),
        # The headline run: Sedov on a jittered mesh, plain FP64.
        dict(_case("sedov", 128, 128, 128, 30, 60), name="Sedov 128^3"),
        # The same in the mixed precision form.
        dict(_case("sedov", 128, 128, 128, 30, 60, precision="mixed"), name="Sedov 128^3 mixed"),
        # An ordinary box whose sides fit nothing, second order with vanLeer.
        dict(_case("sod", 211, 97, 61, 30, 40, limiter="vanLeer"), name="Sod 211x97x61 vanLeer"),
        # The third-order remap with a limiter for uneven widths, its accuracy options in FP64.
        dict(_case("sedov", 90, 75, 66, 20, 40, order=3, limiter="vanLeerG"), name="Sedov 90x75x66 order 3"),
        # Two gases with a perturbed interface: mixed cells, volume fractions among the outputs.
        dict(_case("two gases", 256, 128, 128, 20, 20, fractions=True), name="two gases 256x128x128"),
        # The large production mesh, two gases in the mixed precision form.
        dict(_case("two gases", 384, 384, 192, 12, 8, precision="mixed"), name="two gases 384x384x192 mixed"),
        # A sweep over initial states: uneven meshes advanced together, each with its own dt.
        dict(_case("batch", 32, 96, 0, 20, 20, instances=24), name="batch 24 of 32^3..96^3"),
        dict(_case("batch", 32, 96, 0, 20, 20, instances=24, precision="mixed"), name="batch 24 of 32^3..96^3 mixed"),
    ]


def draw(rng):
    problem = rng.choice(["dt", "sod", "sod", "sedov", "sedov", "two gases", "two gases", "batch"])
    if problem == "batch":
        lo = rng.randint(10, 40)
        return _case("batch", lo, lo + rng.randint(0, 48), 0, rng.randint(5, 20), rng.randint(0, 30),
                     instances=rng.randint(2, 24), precision=rng.choice(["fp64", "mixed"]),
                     limiter=rng.choice(["minmod", "superBee", "vanLeer"]))
    side = 5.0 * 32.0 ** rng.random()                     # 5 .. 160 cells a side on average
    stretch = [2.0 ** (1.2 * rng.random() - 0.6) for _ in range(2)]
    n = [max(3, round(side * s)) for s in (stretch[0], stretch[1], 1.0 / (stretch[0] * stretch[1]))]
    if problem == "dt":
        return _case("dt", *n, 1, 0)
    options = {"precision": rng.choice(["fp64", "fp64", "mixed"]), "order": rng.choice([2, 2, 2, 1]),
               "limiter": rng.choice(["minmod", "superBee", "vanLeer"]), "drive": rng.choice(["step", "entry points"])}
    if options["precision"] == "fp64" and options["order"] == 2:
        extra = rng.choice(["", "", "", "G", "order 3", "csts", "pente-borne", "total energy"])
        if extra == "G":
            options["limiter"] = rng.choice(["minmodG", "superBeeG", "vanLeerG"])
        elif extra == "order 3":
            options["order"] = 3
        elif extra:
            options[{"csts": "csts", "pente-borne": "pente_borne", "total energy": "total_energy"}[extra]] = True
    if problem == "two gases":
        options["fractions"] = rng.random() < 0.5
    return _case(problem, *n, rng.randint(5, 30), rng.randint(10, 50), **options)


# ---- inputs -----------------------------------------------------------------------------------------------------

def _nodes(nx, ny, nz, lengths, jitter, g):
    """The Cartesian mesh, its inner nodes moved by uniform noise of `jitter` cell widths."""
    ax = [torch.arange(n + 1, dtype=torch.float64, device="cuda") * (l / n) for n, l in zip((nx, ny, nz), lengths)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    xyz = torch.stack([x, y, z], dim=3)
    if jitter:
        move = torch.rand(nz - 1, ny - 1, nx - 1, 3, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
        width = torch.tensor([l / n for n, l in zip((nx, ny, nz), lengths)], dtype=torch.float64, device="cuda")
        xyz[1:-1, 1:-1, 1:-1] += move * width * jitter
    return xyz.reshape(-1, 3)


def _options(case, dt):
    return gen.Options(final_time=1e9, deltat_min=0.0, deltat_init=dt, precision=int(case["precision"] == "mixed"),
                       ordre_projection=case["order"], projection_limiteur_id=LIMITERS[case["limiter"]],
                       schema_csts=int(case["csts"]), pente_borne=int(case["pente_borne"]),
                       pente_borne_debar_fix=1, conservation_energie_totale=int(case["total_energy"]))


def _problem(case, problem, nx, ny, nz, g):
    """One mesh with its initial state, as gen.Case."""
    def number(lo, hi):
        return lo + (hi - lo) * float(torch.rand((), generator=g, dtype=torch.float64, device="cuda"))

    C = nx * ny * nz
    longest = max(nx, ny, nz)
    lengths = [n / longest for n in (nx, ny, nz)]
    f64 = dict(dtype=torch.float64, device="cuda")
    if problem == "sod":
        xyz = _nodes(nx, ny, nz, lengths, 0.01, g)
        left = torch.arange(nx, device="cuda").expand(nz, ny, nx).reshape(1, C) < nx // 2
        ratio = math.exp(number(math.log(2.0), math.log(20.0)))
        rho = torch.where(left, 1.0, 1.0 / ratio).to(torch.float64)
        p = torch.where(left, 1.0, 0.1).to(torch.float64)
        gamma, f = [number(1.3, 1.7)], torch.ones(1, C, **f64)
    elif problem == "sedov":
        xyz = _nodes(nx, ny, nz, lengths, 0.01, g)
        e = torch.full((nz, ny, nx), 1e-12, **f64)
        e[:2, :2, :2] = number(0.5, 1.0) / 8.0 * longest ** 3
        gamma, f = [number(1.3, 1.7)], torch.ones(1, C, **f64)
        rho = torch.ones(1, C, **f64)
        p = (gamma[0] - 1.0) * e.reshape(1, C)
    else:
        # x < interface(y, z) is gas A; fractions by 4^3 points a cell
        xyz = _nodes(nx, ny, nz, lengths, 0.0, g)
        ph = torch.rand(4, 2, generator=g, **f64) * (2.0 * math.pi)
        at = [((torch.arange(n * 4, **f64) + 0.5) / (n * 4)) for n in (nx, ny, nz)]
        xi = sum(0.005 * torch.sin(2 * math.pi * m * at[1] + ph[m - 1, 0])[None, :]
                 * torch.sin(2 * math.pi * m * at[2] + ph[m - 1, 1])[:, None] for m in range(1, 5)) + 0.5
        xi = xi.reshape(nz, 4, ny, 4).permute(0, 2, 1, 3).reshape(nz, ny, 1, 16)
        a = torch.zeros(nz, ny, nx, **f64)
        for s in range(4):
            for t in range(16):
                a += at[0][s::4] < xi[..., t]
        a = (a / 64.0).reshape(C)
        f = torch.stack([a, 1.0 - a])
        rho = torch.stack([(a > 0) * 1.0, (a < 1) * 0.2]).to(torch.float64)
        p = torch.stack([(a > 0) * 1.0, (a < 1) * 0.1]).to(torch.float64)
        gamma = [1.4, number(1.5, 1.7)]
    host = [t.cpu().numpy() for t in (xyz, f, rho, p)]
    return gen.Case(problem, nx, ny, nz, host[0], np.array(gamma), host[1], host[2], host[3], np.zeros_like(host[0]),
                    _options(case, 1e-5 if problem == "sedov" else 0.1 / longest), case["cycles"])


def _problems(case, seed):
    g = torch.Generator("cuda").manual_seed(int(seed))
    if case["problem"] != "batch":
        return [_problem(case, case["problem"], case["nx"], case["ny"], case["nz"], g)]
    u = np.random.RandomState(case["nx"] * 1000 + case["ny"]).random_sample(case["instances"])   # the sides
    sides = [case["nx"] + int(x * (case["ny"] - case["nx"] + 1)) for x in u]
    return [_problem(case, ("sod", "sedov")[i % 2], s, s, s, g) for i, s in enumerate(sides)]


def _dt_fields(case, seed):
    g = torch.Generator("cuda").manual_seed(int(seed))
    C, N = case["nx"] * case["ny"] * case["nz"], (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    f64 = dict(dtype=torch.float64, device="cuda", generator=g)
    length = (0.9 + 0.2 * torch.rand(C, **f64)) / case["nx"]
    return length, 1.0 + torch.rand(C, **f64), torch.randn(3, N, **f64)


def prepare(case, seed):
    if case["problem"] == "dt":
        return {"case": case, "fields": _dt_fields(case, seed), "out": torch.empty(2, dtype=torch.float64, device="cuda")}
    problems = _problems(case, seed)
    sim = Batch(problems) if case["problem"] == "batch" else Context(problems[0])
    sim.step(case["lead"])
    sim.synchronize()
    # one pinned buffer a field, the instances of a batch one after the other
    C, N = [p.ncells for p in problems], [p.nnodes for p in problems]
    out, parts = {}, {}
    for name in FIELDS + (("fractions",) if case["fractions"] else ()):
        sizes = [3 * n for n in N] if name == "velocity" else C
        out[name] = torch.empty(sum(sizes), dtype=torch.float64, pin_memory=True)
        parts[name] = out[name].split(sizes)
    return {"case": case, "sim": sim, "out": out, "parts": parts}


# ---- one pass ---------------------------------------------------------------------------------------------------

def _read(call, *a):
    if call(*a) != 0:
        raise RuntimeError(mhy_b200.load().mhy_last_error().decode())


def run(state):
    lib, case = mhy_b200.load(), state["case"]
    if case["problem"] == "dt":
        length, cs, v = state["fields"]
        _read(lib.mhy_compute_hydro_dt_noalloc, case["nx"], case["ny"], case["nz"], length.data_ptr(), cs.data_ptr(),
              v.data_ptr(), 0.3, 1e-3, 0.01, state["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"dt": state["out"]}
    sim, dts = state["sim"], []
    if case["drive"] == "entry points":
        for _ in range(case["cycles"]):
            sim.cycle_by_entry_points()
            dts.append(sim.dt()[0])
    else:
        sim.step(case["cycles"])
    for name, parts in state["parts"].items():
        for i, b in enumerate(parts):
            if case["problem"] == "batch":
                _read(lib.mhy_batch_get_field, sim.h, i, mhy_b200.FIELDS[name], b.data_ptr(), b.numel() * 8)
            elif name == "fractions":
                _read(lib.mhy_get_env_field, sim.h, mhy_b200.ENV_FIELDS["fracvol"], 0, b.data_ptr(), b.numel() * 8)
            else:
                _read(lib.mhy_get_field, sim.h, mhy_b200.FIELDS[name], b.data_ptr(), b.numel() * 8)
    if case["problem"] == "batch":
        dts = [sim.dt(i)[0] for i in range(sim.size())]
    return {"dt": dts or [sim.dt()[0]], **state["out"]}


def work(case):
    """Per cycle the state in and out once: six values a cell (density, energy, pseudo-viscosity, pressure, sound
    speed, mass); per node the velocity, mass and Lagrangian coordinates, and the initial coordinates read; with
    several gases the membership and the fractions too.  Operations of the algorithm as the reference writes it."""
    if case["problem"] == "batch":
        u = np.random.RandomState(case["nx"] * 1000 + case["ny"]).random_sample(case["instances"])
        sizes = [(case["nx"] + int(x * (case["ny"] - case["nx"] + 1)),) * 3 for x in u]
    else:
        sizes = [(case["nx"], case["ny"], case["nz"])]
    C = sum(x * y * z for x, y, z in sizes)
    N = sum((x + 1) * (y + 1) * (z + 1) for x, y, z in sizes)
    if case["problem"] == "dt":
        return {"bytes": 16 * C + 24 * N, "flops": 12 * C + 6 * N}
    gases = 2 if case["problem"] == "two gases" else 1
    cell, node = 2 * 48 + (40 if gases > 1 else 0), 2 * 56 + 24
    read_back = 24 * C + 24 * N + (8 * C if case["fractions"] else 0)
    return {"bytes": case["cycles"] * (cell * C + node * N) + read_back,
            "flops": case["cycles"] * (C * (1300 + 3 * 130 * (3 * gases + 1) / 4) + N * (80 + 3 * 150))}


# ---- what a pass gives, in 64 bits ------------------------------------------------------------------------------
# One perfect gas, order 1 or 2, on the GPU with torch operations: the staggered Lagrange step, the three directional
# remap sweeps of cells and of the dual mesh, the equation of state and the CFL time step.  Arrays are [z, y, x].

CORNERS = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))   # x, y, z offsets
HEX_FACES = ((0, 3, 2, 1), (0, 4, 7, 3), (0, 1, 5, 4), (4, 5, 6, 7), (1, 2, 6, 5), (2, 3, 7, 6))


def _corners(a):
    """The 8 nodal values around each cell, of a [..., z, y, x] array of nodes."""
    n = a.shape[-1] - 1, a.shape[-2] - 1, a.shape[-3] - 1
    return [a[..., k:k + n[2], j:j + n[1], i:i + n[0]] for i, j, k in CORNERS]


def _to_nodes(parts):
    """Sum over the cells around each node: parts[a] is what a cell gives to its corner a."""
    s = list(parts[0].shape)
    out = torch.zeros(s[:-3] + [s[-3] + 1, s[-2] + 1, s[-1] + 1], dtype=torch.float64, device=parts[0].device)
    for (i, j, k), p in zip(CORNERS, parts):
        out[..., k:k + s[-3], j:j + s[-2], i:i + s[-1]] += p
    return out


def _corner_vectors(x):
    """Each corner's area vector: half the triangles that its faces' centres span, 5/12 of the near, 1/12 of the far."""
    near, far = [0.0] * 8, [0.0] * 8
    for face in HEX_FACES:
        centre = sum(x[a] for a in face) / 4
        for m in range(4):
            a, b = face[m], face[(m + 1) % 4]
            t = 0.5 * torch.cross(x[a] - centre, x[b] - centre, dim=0)
            for c in face:
                if c in (a, b):
                    near[c] = near[c] + t
                else:
                    far[c] = far[c] + t
    return [(5.0 * n + f) / 12.0 for n, f in zip(near, far)]


def _cut(a, d, lo, hi):
    return a.narrow(a.dim() - 1 - d, lo, hi - lo)


def _limit(limiter, r):
    if limiter == "minmod":
        return r.clamp(0.0, 1.0)
    if limiter == "superBee":
        return torch.maximum(torch.minimum(2 * r, torch.ones_like(r)), torch.minimum(r, torch.full_like(r, 2.0))).clamp(min=0.0)
    return torch.where(r <= 0, torch.zeros_like(r), 2 * r / (1 + r))


def _slope(limiter, back, front):
    """0.5 (phi(front/back) back + phi(back/front) front), a zero difference contributing nothing."""
    one = torch.ones_like(back)
    b, f = torch.where(back == 0, one, back), torch.where(front == 0, one, front)
    return 0.5 * (torch.where(back == 0, 0.0, _limit(limiter, front / b) * back)
                  + torch.where(front == 0, 0.0, _limit(limiter, back / f) * front))


class _Exact:
    def __init__(self, p, limiter, order):
        shape = (p.nz, p.ny, p.nx)
        nodes = tuple(n + 1 for n in shape)
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        self.gamma, self.limiter, self.o2 = float(p.gamma[0]), limiter, float(order - 1)
        self.x0 = up(p.coords.T).reshape(3, *nodes)
        self.rho, self.p = up(p.density).reshape(shape), up(p.pressure).reshape(shape)
        self.e = self.p / ((self.gamma - 1) * self.rho)
        self.cs, self.q = (self.gamma * self.p / self.rho).sqrt(), torch.zeros_like(self.rho)
        x = _corners(self.x0)
        self.cqs = _corner_vectors(x)
        self.V0 = sum((a * b).sum(0) for a, b in zip(x, self.cqs)) / 3
        self.mass = self.rho * self.V0
        self.nm = _to_nodes([self.mass] * 8) / 8
        self.v, self.Gd = torch.zeros_like(self.x0), torch.zeros_like(self.x0)
        self.dt, self.old_dt, self.turn = p.options.deltat_init, 0.0, 0
        xc = sum(x) / 8
        self.n0, self.out = [], []
        for d in range(3):
            c = self._face_corners(self.x0, d)
            normal = torch.cross(c[2] - c[0], c[3] - c[1], dim=0)
            normal[1] *= -1.0                            # the reference's normal: its y component is turned round
            self.n0.append(normal / normal.norm(dim=0))
            xf, n = sum(c) / 4, shape[2 - d]
            outward = []
            for side in (0, 1):                          # the low and the high face of each cell
                w = _cut(xf, d, side, side + n) - xc
                outward.append(w[d] / w.norm(dim=0))
            self.out.append(outward)

    @staticmethod
    def _face_corners(a, d):
        """The four nodes of each face across d, round the face."""
        o = [ax for ax in range(3) if ax != d]
        got = []
        for s, t in ((0, 0), (1, 0), (1, 1), (0, 1)):
            b = _cut(a, o[0], s, a.shape[a.dim() - 1 - o[0]] - 1 + s)
            got.append(_cut(b, o[1], t, b.shape[b.dim() - 1 - o[1]] - 1 + t))
        return got

    def cycle(self):
        dt = self.dt
        force = _to_nodes([(self.p + self.q) * c for c in self.cqs])
        vh = self.v + 0.5 * (self.old_dt + dt) / self.nm * force
        for d in range(3):
            _cut(vh[d], d, 0, 1).zero_()
            _cut(vh[d], d, vh[d].shape[2 - d] - 1, vh[d].shape[2 - d]).zero_()
        xn = self.x0 + dt * vh
        x = _corners(xn)
        xc = sum(x) / 8
        self.cqs = _corner_vectors(x)
        V = sum((a * b).sum(0) for a, b in zip(x, self.cqs)) / 3
        L = V ** (1.0 / 3.0)
        rho = self.mass / V
        change = 1 / rho - 1 / self.rho
        tau = 0.5 * (1 / self.rho + 1 / rho)
        div = change / dt / tau
        g = self.gamma
        q = torch.where(div < 0, (-0.5 * L * self.cs * div + (g + 1) / 2 * L * L * div * div) / tau, 0.0)
        push = torch.where(q * change < 0, q, 0.0)
        e = (self.e - (0.5 * self.p + push) * change) / (1 + 0.5 * (g - 1) * rho * change)
        self.remap([V, V * rho, V * rho * e, V * q], xn, xc, vh, dt)
        speed = torch.stack(_corners(self.v.norm(dim=0))).amax(0)
        least = float((L / (self.cs + speed)).min())
        self.old_dt, self.dt = dt, min(0.3 * least, 1.05 * dt, 0.01)

    def remap(self, U, xn, xc, vh, dt):
        faces = []
        for d in range(3):
            n = xc.shape[3 - d]
            c = [_cut(t, d, 1, n) for t in self._face_corners(xn, d)]        # inner faces
            n0, xf = _cut(self.n0[d], d, 1, n), sum(c) / 4
            area = 0.5 * torch.cross(c[2] - c[0], c[3] - c[1], dim=0)[d].abs()
            area = torch.where(n0[d].abs() >= 1e-10, area, 0.0)
            u = (sum(_cut(t, d, 1, n) for t in self._face_corners(vh, d)) / 4 * n0).sum(0)
            lo, hi = _cut(xc, d, 0, n - 1), _cut(xc, d, 1, n)
            faces.append((area, u, ((xf - lo) * n0).sum(0), ((xf - hi) * n0).sum(0), ((hi - lo) * n0).sum(0)))
        half_v = 0.5 * vh.norm(dim=0)
        ud = [self.nm * vh[0], self.nm * vh[1], self.nm * vh[2], self.nm, self.nm * half_v]
        P = [vh[0], vh[1], vh[2], half_v]
        for d in [(i + self.turn) % 3 for i in range(3)]:
            n = xc.shape[3 - d]
            area, u, from_lo, from_hi, dx = faces[d]
            phi = [torch.ones_like(U[0])] + [w / U[0] for w in U[1:]]
            back = u * dx > 0
            new = []
            for w, f in zip(U, phi):
                step = (_cut(f, d, 1, n) - _cut(f, d, 0, n - 1)) / dx
                end = torch.zeros_like(_cut(f, d, 0, 1))
                slope = _slope(self.limiter, torch.cat([end, step], 2 - d), torch.cat([step, end], 2 - d)) * (self.o2 > 0)
                value = torch.where(back, _cut(f, d, 0, n - 1) + self.o2 * from_lo * _cut(slope, d, 0, n - 1),
                                    _cut(f, d, 1, n) + self.o2 * from_hi * _cut(slope, d, 1, n))
                through = u * area * dt * value
                low = torch.cat([end, through], 2 - d) * self.out[d][0]
                high = torch.cat([through, end], 2 - d) * self.out[d][1]
                new.append(w - (low + high))
                if w is U[1]:
                    moved = 0.5 * (low * self.out[d][0] + high * self.out[d][1])
            U = [new[0], new[1].clamp(min=0.0), new[2].clamp(min=0.0), new[3]]
            ud, P = self.dual(d, ud, P, xn[d], moved, dt)
        self.rho, self.q = U[1] / self.V0, U[3] / self.V0
        self.e = U[2] / U[1]
        self.mass = U[1]
        self.p = (self.gamma - 1) * self.rho * self.e
        self.cs = (self.gamma * self.p / self.rho).sqrt()
        self.v = torch.stack([w / ud[3] for w in ud[:3]])
        self.nm = _to_nodes([self.mass] * 8) / 8
        self.turn = (self.turn + 1) % 3

    def dual(self, d, ud, P, x, moved, dt):
        """The momentum's remap along d: `moved` is the mass that crossed each cell, the dual faces are the cells."""
        o = [ax for ax in range(3) if ax != d]
        wide = moved
        for ax in o:                                      # a quarter of the four cells round each dual face
            zero = torch.zeros_like(_cut(wide, ax, 0, 1))
            wide = torch.cat([zero, wide], 2 - ax) + torch.cat([wide, zero], 2 - ax)
        m = 0.25 * wide
        n = m.shape[2 - d]                                # cells along d; nodes 1 .. n - 1 are inner
        if self.o2 > 0:
            for c in range(3):
                slope = (_cut(P[c], d, 1, n + 1) - _cut(P[c], d, 0, n)) / (_cut(x, d, 1, n + 1) - _cut(x, d, 0, n))
                _cut(self.Gd[c], d, 1, n).copy_(_slope(self.limiter, _cut(slope, d, 0, n - 1), _cut(slope, d, 1, n)))
        G = [self.Gd[0], self.Gd[1], self.Gd[2], torch.zeros_like(P[3])]
        at = lambda a, s: _cut(a, d, s, n - 1 + s)  # noqa: E731
        mb, mf = at(m, 0), at(m, 1)
        front = at(P[d], 1)
        backward = 0.5 * (at(P[d], 0) + at(P[d], 1))
        sign = lambda w: torch.where(w > 0, 1.0, -1.0)  # noqa: E731
        tf = sign(front) * (at(x, 2) - at(x, 1)) - dt * front
        tb = sign(backward) * (at(x, 1) - at(x, 0)) - dt * backward
        out, phi = [w.clone() for w in ud], []
        for c, slot in enumerate((0, 1, 2, 4)):
            ahead = torch.where(mf < 0, at(P[c], 2) + self.o2 * 0.5 * at(G[c], 2) * tf,
                                at(P[c], 1) + self.o2 * 0.5 * at(G[c], 1) * tf)
            behind = torch.where(mb > 0, at(P[c], 0) + self.o2 * 0.5 * at(G[c], 0) * tb,
                                 at(P[c], 1) + self.o2 * 0.5 * at(G[c], 1) * tb)
            at(out[slot], 1).copy_(at(ud[slot], 1) + (mb * behind - mf * ahead))
        at(out[3], 1).copy_(at(ud[3], 1) + (mb - mf))
        for c, slot in enumerate((0, 1, 2, 4)):
            f = P[c].clone()
            at(f, 1).copy_(at(out[slot], 1) / at(out[3], 1))
            phi.append(f)
        return out, phi


def exact(case, seed):
    """None for what has no short independent form: several gases, order 3, the uneven-width limiters, csts,
    pente-borne, the total-energy option."""
    if case["problem"] == "dt":
        length, cs, v = _dt_fields(case, seed)
        speed = torch.stack(_corners(v.norm(dim=0).reshape(case["nz"] + 1, case["ny"] + 1, case["nx"] + 1))).amax(0)
        least = (length / (cs + speed.reshape(-1))).min()
        return {"dt": torch.stack([least, torch.clamp(0.3 * least, max=1.05e-3)])}
    if (case["problem"] == "two gases" or case["order"] == 3 or LIMITERS[case["limiter"]] >= 3 or case["csts"]
            or case["pente_borne"] or case["total_energy"]):
        return None
    got = []
    for p in _problems(case, seed):
        e = _Exact(p, case["limiter"], case["order"])
        dts = []
        for i in range(case["lead"] + case["cycles"]):
            e.cycle()
            dts.append(e.dt)
        got.append({"dt": dts[case["lead"]:] if case["drive"] == "entry points" else dts[-1:], "density": e.rho.reshape(-1),
                    "internal_energy": e.e.reshape(-1), "pressure": e.p.reshape(-1),
                    "velocity": e.v.reshape(3, -1).T.reshape(-1)})
        del e
    if case["problem"] == "batch":
        return {"dt": [o["dt"][-1] for o in got],
                **{name: torch.cat([o[name] for o in got]) for name in FIELDS}}
    return got[0]
