"""The workloads this framework's speed is measured on.

Every case is a call (or a short sequence of calls) a user's program makes:
set a wavefunction on a solver, step it, read it back; a sweep of independent
solves; a served stream of requests; the analysis of a resident state.  Units
are hbar = m = 1.  A case is a dict of plain values:

  kind "evolve"   one Solver: wavefunction in, `steps` split-operator steps with
                  an energy check every `check` steps (0: none), wavefunction out
  kind "batch"    `solves` 2D ground-state solves of uneven sizes as one Batch
  kind "serve"    `requests` solves of mixed sizes through a resident Server
  kind "analyse"  vortex finder and observables of a resident 2D state

precision "f64" is the plain complex128 form, "f32" the fused complex64 form;
time "imag" relaxes to the ground state, "real" follows the dynamics.
"""

import math
import random

import numpy as np
import torch

import gpue_b200 as G

# lengths with a compiled transform
LENGTHS = (16, 32, 64, 96, 128, 160, 192, 256, 320, 384, 512, 640, 768, 1024)
LENGTHS_3D = (32, 64, 96, 128, 160, 192, 256)
SWEEP_LENGTHS = (128, 192, 256, 384, 512)
DT_IMAG, DT_REAL = 1e-4, 5e-5
# static potential of a parameter file: the harmonic trap plus a square lattice
LATTICE_DEPTH, LATTICE_K = 25.0, 2.5
LATTICE_TEXT = ("V = 0.5*mass*((omegaX*x)*(omegaX*x)+(omegaY*y)*(omegaY*y))"
                "+%g*(cos(%g*x)*cos(%g*x)+cos(%g*y)*cos(%g*y))"
                % (LATTICE_DEPTH, LATTICE_K, LATTICE_K, LATTICE_K, LATTICE_K))
OBSERVABLES = ("norm", "energy", "e_kinetic", "e_potential", "e_interaction", "e_rotation",
               "x", "y", "z", "r2", "q", "lz")


def evolve(name, dim, n, precision, time, steps, check=0, omega=0.0, g=100.0, wz=1.0,
           box=10.0, field="trap"):
    return {"name": name, "kind": "evolve", "dim": dim, "n": n, "precision": precision,
            "time": time, "steps": steps, "check": check, "omega": omega, "g": g, "wz": wz,
            "box": box, "field": field}


def listed():
    return [
        # a short relaxation of a tiny grid, as a test or a parameter scan makes them:
        # latency and launches
        evolve("relax2d_64_f64", 2, 64, "f64", "imag", 10, g=50.0, box=8.0),
        # the plain 256^2 ground state with its energy checks (a slice of 10,000 steps)
        evolve("ground2d_256_f64", 2, 256, "f64", "imag", 200, check=100),
        # rotating-frame dynamics in double precision on a radix-3 grid
        evolve("rotate2d_384_f64", 2, 384, "f64", "real", 60, omega=0.6, g=300.0, box=12.0),
        # the 1024^2 rotating condensate in the complex64 form (a slice of 20,000 steps)
        evolve("rotate2d_1024_f32", 2, 1024, "f32", "real", 100, omega=0.7, g=500.0, box=16.0),
        # a potential given as a full field (parameter file) instead of the trap
        evolve("lattice2d_512_f64", 2, 512, "f64", "imag", 50, check=25, g=200.0,
               field="lattice"),
        # the largest ground state, anisotropic trap, in both forms
        evolve("ground3d_256_f32", 3, 256, "f32", "imag", 21, check=10, g=1000.0, wz=4.0,
               box=12.0),
        evolve("ground3d_256_f64", 3, 256, "f64", "imag", 8, g=1000.0, wz=4.0, box=12.0),
        # 3D dynamics without rotation on a radix-5 grid
        evolve("dynamics3d_160_f32", 3, 160, "f32", "real", 40, g=400.0, box=10.0),
        # a rotating 3D ground state (gauge passes) in double precision
        evolve("rotate3d_96_f64", 3, 96, "f64", "imag", 40, omega=0.5, g=200.0, box=9.0),
        # a parameter sweep: independent 2D ground states, uneven sizes, checked every 100
        {"name": "sweep2d_f32", "kind": "batch", "solves": 16, "steps": 201, "check": 100,
         "sizes": 4},
        # a served stream of mixed 2D/3D imaginary- and real-time requests
        {"name": "serve_f32", "kind": "serve", "requests": 10, "steps": 200, "sizes": 5,
         "top2d": 1024, "top3d": 128},
        # print-step analysis of a rotating state: vortices and observables
        {"name": "analyse2d_768_f32", "kind": "analyse", "n": 768, "precision": "f32",
         "omega": 0.7, "box": 14.0},
    ]


def draw(rng):
    kind = rng.choices(("evolve", "batch", "serve", "analyse"), (8, 1, 1, 1))[0]
    if kind == "batch":
        return {"kind": "batch", "solves": rng.randint(3, 20),
                "steps": 50 * rng.randint(1, 3) + 1, "check": 50, "sizes": rng.randrange(1 << 20)}
    if kind == "serve":
        return {"kind": "serve", "requests": rng.randint(2, 10),
                "steps": 100 * rng.randint(1, 2), "sizes": rng.randrange(1 << 20),
                "top2d": rng.choice((512, 768, 1024)), "top3d": rng.choice((64, 96, 128))}
    if kind == "analyse":
        return {"kind": "analyse", "n": rng.choice(LENGTHS[2:]),
                "precision": rng.choice(("f32", "f64")), "omega": round(rng.uniform(0, 0.8), 3),
                "box": round(rng.uniform(8, 16), 2)}
    dim = rng.choice((2, 2, 3))
    precision = rng.choice(("f64", "f32"))
    n = rng.choice(LENGTHS if dim == 2 else LENGTHS_3D)
    most = 4e9 / (n ** dim * (32 if precision == "f64" else 16))
    most = max(5.0, min(200.0, most))
    steps = int(round(math.exp(rng.uniform(math.log(5.0), math.log(most)))))
    c = evolve("", dim, n, precision, rng.choice(("imag", "real")), steps,
               check=rng.choice((0, 0, max(1, steps // 2))),
               omega=rng.choice((0.0, 0.0, round(rng.uniform(0.1, 0.8), 3))),
               g=round(math.exp(rng.uniform(math.log(10.0), math.log(1000.0))), 2),
               wz=rng.choice((1.0, 4.0)) if dim == 3 else 1.0,
               box=round(rng.uniform(8.0, 14.0), 2))
    if dim == 2 and c["omega"] == 0.0 and rng.random() < 0.25:
        c["field"] = "lattice"
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs --

def grid(n, box):
    dx = box / (n >> 1)
    return -box + dx * torch.arange(n, dtype=torch.float64, device="cuda"), dx


def momenta(n, box):
    return torch.fft.fftfreq(n, d=1.0 / n, dtype=torch.float64, device="cuda") * (math.pi / box)


def along(v, axis, dim):
    """A per-axis vector shaped to broadcast over [z, y, x] (axis 0 = x)."""
    shape = [1] * dim
    shape[dim - 1 - axis] = v.numel()
    return v.reshape(shape)


def start_state(dim, n, box, real_time, seed):
    """A Gaussian cloud with 1 % noise; for dynamics and analysis times a smoothed random
    phase (correlation length 1/20 of the box), which holds vortices.  complex128,
    sum |psi|^2 dV = 1."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    x, dx = grid(n, box)
    r2 = sum(along(x, a, dim) ** 2 for a in range(dim))
    width = box / 4.5
    noise = torch.randn((n,) * dim, generator=gen, dtype=torch.float64, device="cuda")
    psi = (torch.exp(-r2 / (2 * width * width)) * (1.0 + 0.01 * noise)).to(torch.complex128)
    if real_time:
        th = torch.randn((n,) * dim, generator=gen, dtype=torch.float64, device="cuda")
        k2 = sum(along(momenta(n, box), a, dim) ** 2 for a in range(dim))
        th = torch.fft.ifftn(torch.fft.fftn(th) * torch.exp(-0.5 * k2 * (box / 20) ** 2)).real
        psi = psi * torch.exp(2j * th / th.std())
    return psi / torch.sqrt(torch.sum(psi.abs() ** 2) * dx ** dim)


def solver(dim, n, box, precision, g, omega, wy=1.0, wz=1.0, gdt=DT_IMAG, dt=DT_REAL):
    return G.Solver(params(dim, n, box, precision, g, omega, wy, wz, gdt, dt))


def params(dim, n, box, precision, g, omega, wy=1.0, wz=1.0, gdt=DT_IMAG, dt=DT_REAL):
    return G.make_params(dim, n, box, wy=wy, wz=wz, g=g, omega=omega, gauge=omega != 0.0,
                         gdt=gdt, dt=dt,
                         precision=G.PREC_FP32 if precision == "f32" else G.PREC_FP64)


def stored(psi, precision):
    return psi.to(torch.complex64) if precision == "f32" else psi


def code(precision):
    return G.C64 if precision == "f32" else G.C128


def sweep_solves(case, seed):
    """The solves of a batch case: sizes by the case, physics and states by the seed."""
    by_size, by_seed = random.Random(case["sizes"]), random.Random(seed)
    return [{"n": by_size.choice(SWEEP_LENGTHS), "g": by_seed.uniform(10.0, 1000.0),
             "wy": by_seed.uniform(0.8, 1.25), "seed": seed * 100 + k}
            for k in range(case["solves"])]


def serve_requests(case, seed):
    """The requests of a serve case: 70 % 2D and 30 % 3D, half of them in real time with a
    rotation; sizes and kinds by the case, physics and states by the seed."""
    by_size, by_seed = random.Random(case["sizes"]), random.Random(seed)
    out = []
    for k in range(case["requests"]):
        dim = 2 if by_size.random() < 0.7 else 3
        n = by_size.choice([m for m in LENGTHS if (128 if dim == 2 else 64) <= m
                            <= (case["top2d"] if dim == 2 else case["top3d"])])
        real = by_size.random() < 0.5
        out.append({"dim": dim, "n": n, "real": real, "box": 10.0 if dim == 2 else 8.0,
                    "g": by_seed.uniform(10.0, 1000.0),
                    "omega": by_seed.uniform(0.1, 0.8) if real else 0.0, "seed": seed * 100 + k})
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "evolve":
        dim, n, box, prec = case["dim"], case["n"], case["box"], case["precision"]
        s = solver(dim, n, box, prec, case["g"], case["omega"], wz=case["wz"])
        if case["field"] == "lattice":
            s.load_param_text(LATTICE_TEXT)
        psi = stored(start_state(dim, n, box, case["time"] == "real", seed), prec)
        gstate = 1 if case["time"] == "real" else 0
        s.set_operators(gstate)
        return {"kind": kind, "solver": s, "psi": psi, "out": torch.empty_like(psi),
                "dtype": code(prec), "gstate": gstate, "steps": case["steps"],
                "check": case["check"], "f32": prec == "f32"}
    if kind == "batch":
        solves = sweep_solves(case, seed)
        ss = [solver(2, q["n"], 10.0, "f32", q["g"], 0.0, wy=q["wy"]) for q in solves]
        psi = [stored(start_state(2, q["n"], 10.0, False, q["seed"]), "f32") for q in solves]
        return {"kind": kind, "solvers": ss, "batch": G.Batch(ss), "psi": psi,
                "out": [torch.empty_like(p) for p in psi], "steps": case["steps"],
                "check": case["check"]}
    if kind == "serve":
        reqs = serve_requests(case, seed)
        jobs = [(params(q["dim"], q["n"], q["box"], "f32", q["g"], q["omega"]),
                 1 if q["real"] else 0,
                 start_state(q["dim"], q["n"], q["box"], q["real"], q["seed"]).cpu().numpy())
                for q in reqs]
        server = G.Server(precision=G.PREC_FP32, check_steps=100, threshold=0.0)
        return {"kind": kind, "server": server, "jobs": jobs, "steps": case["steps"]}
    n, box, prec = case["n"], case["box"], case["precision"]
    s = solver(2, n, box, prec, 500.0, case["omega"])
    psi = stored(start_state(2, n, box, True, seed), prec)
    s.set_operators(1)
    s.set_wfc_device(psi.data_ptr(), code(prec))
    return {"kind": kind, "solver": s, "radius": 0.5 * box, "f32": prec == "f32"}


# --------------------------------------------------------------------- run --

def run(state):
    return {"evolve": run_evolve, "batch": run_batch, "serve": run_serve,
            "analyse": run_analyse}[state["kind"]](state)


def run_evolve(st):
    s = st["solver"]
    s.set_wfc_device(st["psi"].data_ptr(), st["dtype"])
    r = s.evolve(st["steps"], st["gstate"], energy_every=st["check"])
    s.get_wfc_device(st["out"].data_ptr(), st["dtype"])
    out = {"psi": st["out"]}
    if st["check"]:
        out["energy"] = np.float32(r["energy"]) if st["f32"] else r["energy"]
    return out


def run_batch(st):
    for s, p in zip(st["solvers"], st["psi"]):
        s.set_wfc_device(p.data_ptr(), G.C64)
    res, _ = st["batch"].evolve(0, st["steps"], energy_every=st["check"])
    for s, p in zip(st["solvers"], st["out"]):
        s.get_wfc_device(p.data_ptr(), G.C64)
    return {"psi": st["out"], "energy": np.array([r["energy"] for r in res], dtype=np.float32),
            "steps": [r["steps_done"] for r in res]}


def run_serve(st):
    srv = st["server"]
    for tag, (p, gstate, psi0) in enumerate(st["jobs"]):
        srv.submit(p, gstate, st["steps"], psi0, tag)
    got = {}
    while len(got) < len(st["jobs"]):
        for r in srv.poll(timeout=10.0):
            got[r["tag"]] = r
    got = [got[k] for k in range(len(st["jobs"]))]
    return {"psi": [r["psi"].astype(np.complex64) for r in got],
            "energy": np.array([r["energy"] for r in got], dtype=np.float32),
            "steps": [r["steps_done"] for r in got], "status": [r["status"] for r in got]}


def run_analyse(st):
    s = st["solver"]
    marker, marks, found = s.find_vortices(st["radius"])
    o = s.observables()
    return {"marker": marker, "i": marks["i"], "j": marks["j"], "winding": marks["winding"],
            "found": found,
            "observables": np.array([o[k] for k in OBSERVABLES],
                                    dtype=np.float32 if st["f32"] else np.float64)}


# -------------------------------------------------------------------- work --

def solve_work(dim, n, precision, steps, gauge, field_table=False):
    """One read and one write of the field per step (plus a tabulated potential's read);
    the steps' transforms at 5 n log2 n each way and axis and about 40 operations a point
    for the phase factors."""
    pts = n ** dim
    size = 8 if precision == "f32" else 16
    lines = 2 * dim + (4 if gauge else 0)
    return {"bytes": steps * pts * (2 * size + (8 if field_table else 0)),
            "flops": steps * pts * (lines * 5 * math.log2(n) + 40 + (12 if gauge else 0))}


def work(case):
    kind = case["kind"]
    if kind == "evolve":
        return solve_work(case["dim"], case["n"], case["precision"], case["steps"],
                          case["omega"] != 0.0, case["field"] == "lattice")
    if kind == "analyse":
        pts = case["n"] ** 2
        size = 8 if case["precision"] == "f32" else 16
        return {"bytes": pts * (size + 4), "flops": pts * (10 * math.log2(case["n"]) + 100)}
    if kind == "batch":
        parts = [solve_work(2, q["n"], "f32", case["steps"], False)
                 for q in sweep_solves(case, 0)]
    else:
        parts = [solve_work(q["dim"], q["n"], "f32", case["steps"], q["real"])
                 for q in serve_requests(case, 0)]
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


# ------------------------------------------------------- 64-bit references --

class Exact:
    """The split step in complex128 with torch's transforms."""

    def __init__(self, dim, n, box, g, omega, wy=1.0, wz=1.0, field="trap"):
        self.dim, self.n, self.box, self.g, self.omega = dim, n, box, g, omega
        self.x, self.dx = grid(n, box)
        self.p = momenta(n, box)
        w = (1.0, wy, wz)
        # the rotation gauge A = omega (-wx y, wy x, 0) adds |A|^2/2 to the potential
        self.a = (-omega, omega * wy)
        V = sum(0.5 * (w[k] * along(self.x, k, dim)) ** 2 for k in range(dim))
        if omega:
            V = V + 0.5 * ((self.a[0] * along(self.x, 1, dim)) ** 2 +
                           (self.a[1] * along(self.x, 0, dim)) ** 2)
        if field == "lattice":
            V = V + LATTICE_DEPTH * sum(torch.cos(LATTICE_K * along(self.x, k, dim)) ** 2
                                        for k in range(dim))
        self.V = V.expand((n,) * dim)
        self.K = sum(0.5 * along(self.p, k, dim) ** 2 for k in range(dim))

    def normalise(self, psi):
        return psi / torch.sqrt(torch.sum(psi.abs() ** 2) * self.dx ** self.dim)

    def half(self, psi, z):
        return psi * torch.exp(-z * (self.V + self.g * psi.abs() ** 2))

    def gauge(self, psi, axis, z):
        """exp(-z A_axis p_axis) along one axis (0 = x)."""
        ax = self.dim - 1 - axis
        A = self.a[axis] * along(self.x, 1 - axis, self.dim)
        return torch.fft.ifft(torch.fft.fft(psi, dim=ax) *
                              torch.exp(-z * A * along(self.p, axis, self.dim)), dim=ax)

    def step(self, psi, i, real, dt):
        z = 1j * dt if real else dt
        psi = self.half(psi, 0.5 * z)
        psi = torch.fft.ifftn(torch.fft.fftn(psi) * torch.exp(-z * self.K))
        psi = self.half(psi, 0.5 * z)
        if self.omega:
            for axis in ((0, 1) if i % 2 else (1, 0)):
                psi = self.gauge(psi, axis, z)
        return psi if real else self.normalise(psi)

    def diff(self, psi, axis):
        """Forward difference over the flat index; psi/d past the end."""
        f = psi.reshape(-1)
        s = self.n ** axis
        out = f / self.dx
        out[:-s] = (f[s:] - f[:-s]) / self.dx
        return out.reshape(psi.shape)

    def terms(self, psi):
        dV, d = self.dx ** self.dim, psi.abs() ** 2
        kin = torch.sum(self.K * torch.fft.fftn(psi).abs() ** 2) / psi.numel() * dV
        rot = 0.0
        if self.omega:
            A = [self.a[k] * along(self.x, 1 - k, self.dim) for k in range(2)]
            rot = torch.sum((psi.conj() * 1j * (A[0] * self.diff(psi, 0) +
                                                A[1] * self.diff(psi, 1))).real) * dV
        return [float(t) for t in (kin, torch.sum(self.V * d) * dV,
                                   torch.sum(0.5 * self.g * d * d) * dV, rot)]

    def evolve(self, psi, steps, real, dt, check=0):
        energy = math.nan
        for i in range(steps):
            psi = self.step(psi, i, real, dt)
            if check and i % check == 0:
                energy = sum(self.terms(psi))
        return psi, energy

    def observables(self, psi):
        dV, d = self.dx ** 2, psi.abs() ** 2
        t = self.terms(psi)
        w = torch.ones(self.n, dtype=torch.float64, device="cuda")
        w[0] = w[-1] = 0.5
        wd = d * along(w, 0, 2) * along(w, 1, 2)
        X, Y = along(self.x, 0, 2), along(self.x, 1, 2)
        lz = torch.sum((psi.conj() * -1j * (X * self.diff(psi, 1) - Y * self.diff(psi, 0))).real)
        moments = [torch.sum(wd * m) * dV for m in (X, Y)]
        last = [torch.sum(wd * (X * X + Y * Y)) * dV, torch.sum(wd * (X * X - Y * Y)) * dV,
                lz * dV]
        return np.array([float(v) for v in [torch.sum(d) * dV, sum(t)] + t + moments + [0.0]
                         + last])


def exact(case, seed):
    kind = case["kind"]
    if kind == "evolve":
        prec, real = case["precision"], case["time"] == "real"
        e = Exact(case["dim"], case["n"], case["box"], case["g"], case["omega"], wz=case["wz"],
                  field=case["field"])
        psi = stored(start_state(case["dim"], case["n"], case["box"], real, seed), prec)
        psi, energy = e.evolve(psi.to(torch.complex128), case["steps"], real,
                               DT_REAL if real else DT_IMAG, case["check"])
        return {"psi": psi, "energy": energy} if case["check"] else {"psi": psi}
    if kind == "batch":
        out = {"psi": [], "energy": [], "steps": None}
        for q in sweep_solves(case, seed):
            e = Exact(2, q["n"], 10.0, q["g"], 0.0, wy=q["wy"])
            psi = stored(start_state(2, q["n"], 10.0, False, q["seed"]), "f32")
            psi, energy = e.evolve(psi.to(torch.complex128), case["steps"], False, DT_IMAG,
                                   case["check"])
            out["psi"].append(psi)
            out["energy"].append(energy)
        out["energy"] = np.array(out["energy"])
        return out
    if kind == "serve":
        out = {"psi": [], "energy": [], "steps": None, "status": None}
        for q in serve_requests(case, seed):
            e = Exact(q["dim"], q["n"], q["box"], q["g"], q["omega"])
            psi = start_state(q["dim"], q["n"], q["box"], q["real"], q["seed"])
            psi, _ = e.evolve(psi, case["steps"], q["real"], DT_REAL if q["real"] else DT_IMAG)
            out["psi"].append(psi)
            out["energy"].append(sum(e.terms(psi)))
        out["energy"] = np.array(out["energy"])
        return out
    e = Exact(2, case["n"], case["box"], 500.0, case["omega"])
    psi = stored(start_state(2, case["n"], case["box"], True, seed), case["precision"])
    return {"marker": None, "i": None, "j": None, "winding": None, "found": None,
            "observables": e.observables(psi.to(torch.complex128))}
