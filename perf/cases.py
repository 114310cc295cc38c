"""Performance cases of the library, through its Python front end.

Four kinds of work, each as a user's program has it done:

rollout   a running simulation is advanced by `steps` iterations and its
          state is read into device arrays (the output step of a run).  The
          state carries over from one pass to the next.  The mixed form's
          fields are read as FP32, what they are computed in.
coupled   the particle state lives in a host program (a DEM code, a
          controller): every iteration uploads it, runs one step and reads
          positions and forces back.
gradient  one evaluation of a trajectory's gradient (FP64): set the initial
          state, run forward with checkpoints, run backward from a cotangent
          of the final state, read the gradients.
calls     the fine-grained calls that stand for the reference's field,
          cluster and element functions, on host arrays.

Grids are periodic boxes with dx = 1 (powers of two per axis, as the library
takes them); spheres sit on a jittered lattice, or anywhere (`overlap`) where
the radii do not fit one.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import fipi_gb300 as F
from fipi_gb300.params import REF_PI, Workload

# ------------------------------------------------------------------ cases


def _case(name, kind, precision, nx, ny, nz, n_p, r_p, steps, **more):
    c = {"name": name, "kind": kind, "precision": precision, "nx": nx, "ny": ny, "nz": nz, "n_p": n_p, "r_p": r_p,
         "steps": steps, "phi_mean": 0.0, "rho2": 1e-3, "polydisperse": False, "overlap": False, "conserve": False,
         "couple": False, "dt": 1e-3}
    c.update(more)
    return c


def listed():
    return [
        # The smallest grid of the parity tests: a step is launch latency only.
        _case("rollout_mixed_16", "rollout", "mixed", 16, 16, 16, 6, 1.0, 10),
        # The 64^3 case of the benchmark plan (256 spheres): small studies and
        # parameter sweeps, both forms.
        _case("rollout_mixed_64", "rollout", "mixed", 64, 64, 64, 256, 4.0, 10),
        _case("rollout_fp64_64", "rollout", "fp64", 64, 64, 64, 256, 4.0, 10),
        # A slab-like box with unequal axes, an odd particle count, spread
        # radii, a density contrast and the fluid coupling on.
        _case("rollout_mixed_aniso", "rollout", "mixed", 128, 64, 256, 2999, 3.0, 8, polydisperse=True, rho2=5e-2,
              couple=True),
        # The same kind of box in FP64 in the mass-conserving mode, with long
        # y and z axes and short rows along x.
        _case("rollout_fp64_aniso", "rollout", "fp64", 32, 256, 128, 701, 2.0, 4, phi_mean=-0.2, conserve=True),
        # The headline workload (256^3, 20,000 spheres) in both forms.
        _case("rollout_mixed_256", "rollout", "mixed", 256, 256, 256, 20000, 4.0, 10),
        _case("rollout_fp64_256", "rollout", "fp64", 256, 256, 256, 20000, 4.0, 3),
        # The largest: off-critical quench, 200,000 polydisperse spheres above
        # the jamming limit (overlaps allowed).
        _case("rollout_mixed_512", "rollout", "mixed", 512, 512, 512, 200000, 4.5, 4, phi_mean=-0.4, dt=5e-4,
              polydisperse=True, overlap=True),
        # A host program that owns the particles, 128^3.
        _case("coupled_mixed_128", "coupled", "mixed", 128, 128, 128, 2000, 4.0, 4),
        # Gradients: the parity tests' 32^3 trajectory and the 128^3,
        # 2000-sphere case of the gradient check, a short window of it.
        _case("gradient_fp64_32", "gradient", "fp64", 32, 32, 32, 40, 1.2, 6),
        _case("gradient_fp64_128", "gradient", "fp64", 128, 128, 128, 2000, 4.0, 4),
        # One of each fine-grained call on host arrays.
        _case("calls_fp64_64", "calls", "fp64", 64, 64, 64, 256, 4.0, 1),
    ]


def draw(rng):
    kind = rng.choice(["rollout"] * 6 + ["coupled", "gradient", "gradient", "calls"])
    precision = "fp64" if kind in ("gradient", "calls") else rng.choice(["mixed", "mixed", "fp64"])
    top = {"rollout": 24, "coupled": 22, "gradient": 20, "calls": 19}[kind]  # log2 of the most grid points
    while True:
        e = [rng.randint(4, 9) for _ in range(3)]
        if sum(e) <= top:
            break
    nx, ny, nz = (1 << k for k in e)
    V = nx * ny * nz
    r_p = round(min(4.0, min(nx, ny, nz) / 16.0) * rng.uniform(0.7, 1.0), 3)  # at least 3 cells of 5 r_p per axis
    most = max(3.0, min(30000.0, 60.0 * V / (524.0 * r_p ** 3)))  # up to 60 partners within the contact range
    n_p = 0 if kind == "rollout" and rng.random() < 0.1 else int(round(math.exp(rng.uniform(math.log(3.0), math.log(most)))))
    cost = V * (6.0 if precision == "fp64" else 1.0) * (4.0 if kind == "gradient" else 1.0)
    steps = 1 if kind == "calls" else rng.randint(2, max(2, min(10, int(2.0 ** 28 / cost))))
    return {"kind": kind, "precision": precision, "nx": nx, "ny": ny, "nz": nz, "n_p": max(n_p, 1) if kind != "rollout" else n_p,
            "r_p": r_p, "steps": steps, "phi_mean": rng.choice([0.0, 0.0, -0.4]), "rho2": rng.choice([1e-3, 5e-2]),
            "polydisperse": rng.random() < 0.4, "overlap": rng.random() < 0.2,
            "conserve": kind == "rollout" and rng.random() < 0.2, "couple": kind == "rollout" and rng.random() < 0.2,
            "dt": rng.choice([1e-3, 5e-4])}


# ------------------------------------------------------------------ inputs


def _params(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return Workload("case", nx, ny, nz, float(nx), float(ny), float(nz), n_p=case["n_p"], r_p=case["r_p"],
                    dt=case["dt"], t_end=500, rho2=case["rho2"]).params()


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _phase(case, seed, device):
    """phi = mean + U(-0.05, 0.05), the quench of every workload."""
    g = torch.Generator(device=device).manual_seed(1000 * seed + 1)
    V = case["nx"] * case["ny"] * case["nz"]
    c = torch.rand(V, generator=g, device=device, dtype=torch.float64)
    return c.sub_(0.5).mul_(0.1).add_(case["phi_mean"])


def _particles(case, seed):
    """Positions (n x 3), radii, cos(theta) and contact forces (n x 3)."""
    rng = np.random.default_rng(1000 * seed + 2)
    n = case["n_p"]
    L = np.array([case["nx"], case["ny"], case["nz"]], dtype=np.float64)
    if case["overlap"] or n == 0:
        p = rng.uniform(0.0, 1.0, (n, 3)) * L
    else:
        s = (L.prod() / n) ** (1.0 / 3.0)
        m = np.ceil(L / s).astype(int)
        site = rng.permutation(int(m.prod()))[:n]
        at = np.stack([site % m[0], site // m[0] % m[1], site // (m[0] * m[1])], axis=1)
        p = (at + 0.5 + rng.uniform(-0.15, 0.15, (n, 3))) * (L / m)
    r = np.full(n, case["r_p"])
    ct = np.zeros(n)
    if case["polydisperse"]:
        r = case["r_p"] * rng.uniform(2.0 / 3.0, 4.0 / 3.0, n)
        ct = np.cos(np.radians(rng.uniform(60.0, 120.0, n)))
    f = 0.1 * rng.standard_normal((n, 3))
    return p, r, ct, f


def _normals(shape, seed, k, device):
    g = torch.Generator(device=device).manual_seed(1000 * seed + k)
    return torch.randn(shape, generator=g, device=device, dtype=torch.float64)


def prepare(case, seed):
    P = _params(case)
    V, n = P.nx * P.ny * P.nz, P.n_p
    sim = F.Simulation(P, case["precision"])
    dev = "cuda"
    s = {"case": case, "sim": sim}
    c = _phase(case, seed, dev)
    p, r, ct, f = _particles(case, seed)
    if case["kind"] == "calls":
        s["x"] = c.cpu().numpy()
        s["p"], s["f"] = p.ravel(), f.ravel()
        s["X"] = np.ascontiguousarray(np.fft.rfftn(s["x"].reshape(P.nz, P.ny, P.nx)).transpose(0, 2, 1)).ravel()
        return s
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev).reshape(-1)  # noqa: E731
    torch.cuda.synchronize()
    s["c"] = torch.empty(V, dtype=torch.float64, device=dev)
    s["u"] = torch.empty(3 * V, dtype=torch.float64, device=dev)
    if case["kind"] == "gradient":
        s["c0"], s["p0"], s["r"], s["ct"], s["f0"] = c, put(p), put(r), put(ct), put(f)
        s["u0"] = 0.01 * _normals(3 * V, seed, 3, dev)
        s["dc"] = _normals(V, seed, 4, dev).cpu().numpy()
        s["du"] = _normals(3 * V, seed, 5, dev).cpu().numpy()
        rng = np.random.default_rng(1000 * seed + 6)
        s["dp"], s["df"] = rng.standard_normal(3 * n), rng.standard_normal(3 * n)
        torch.cuda.synchronize()
        return s
    sim.set_phase_device(c)
    if case["conserve"]:
        sim.set_mass_conserving(True)
    if case["couple"]:
        sim.set_fluid_coupling(True)
    if n:
        sim.set_particles(p, r, ct, f)
    sim.sync()
    s["stream"] = torch.cuda.ExternalStream(sim.stream())
    s["out"] = {}
    if case["precision"] == "mixed":
        s["out"] = {"phase": torch.empty(V, dtype=torch.float32, device=dev),
                    "velocity": torch.empty(3 * V, dtype=torch.float32, device=dev)}
    if case["kind"] == "coupled":
        s["p"], s["r"], s["ct"], s["f"] = p.ravel(), r, ct, f.ravel()
        s["got"] = tuple(np.empty(3 * n) for _ in range(3))
        return s
    s["pp"], s["fpp"], s["fpi"] = (torch.empty(3 * n, dtype=torch.float64, device=dev) for _ in range(3))
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ passes


def run(s):
    return {"rollout": _rollout, "coupled": _coupled, "gradient": _gradient, "calls": _calls}[s["case"]["kind"]](s)


def _fields(s):
    """phi and u of the state; the mixed form's as FP32, on the library's stream."""
    sim = s["sim"]
    sim.get_phase_device(s["c"])
    sim.get_velocity_device(s["u"])
    if s["case"]["precision"] != "mixed":
        return {"phase": s["c"], "velocity": s["u"]}
    with torch.cuda.stream(s["stream"]):
        s["out"]["phase"].copy_(s["c"])
        s["out"]["velocity"].copy_(s["u"])
    return dict(s["out"])


def _rollout(s):
    sim = s["sim"]
    sim.step(s["case"]["steps"])
    out = _fields(s)
    if sim.n:
        sim.get_particles_device(s["pp"], s["fpp"], s["fpi"])
        out["positions"] = s["pp"]
        if s["case"]["precision"] == "mixed":
            with torch.cuda.stream(s["stream"]):
                out["f_pp"], out["f_pi"] = s["fpp"].float(), s["fpi"].float()
        else:
            out["f_pp"], out["f_pi"] = s["fpp"], s["fpi"]
    return out


def _coupled(s):
    sim = s["sim"]
    for _ in range(s["case"]["steps"]):
        sim.set_particles(s["p"], s["r"], s["ct"], s["f"])
        sim.step_async(1)
        p, f, _ = sim.get_particles(s["got"])
        s["p"], s["f"] = p.copy(), f.copy()  # what the host program keeps and would move on its own
    out = _fields(s)
    real = np.float32 if s["case"]["precision"] == "mixed" else np.float64
    out["positions"], out["f_pp"], out["f_pi"] = s["p"], s["f"].astype(real), s["got"][2].astype(real)
    return out


def _gradient(s):
    sim = s["sim"]
    sim.set_phase_device(s["c0"])
    sim.set_velocity_device(s["u0"])
    sim.set_particles_device(s["p0"], s["r"], s["ct"], s["f0"])
    sim.trajectory_forward(s["case"]["steps"])
    sim.get_phase_device(s["c"])
    sim.trajectory_backward(s["dc"], s["du"], s["dp"], s["df"])
    dc, du, dp, df = sim.adjoint_get()
    g, dct = sim.adjoint_get_params()
    return {"phase": s["c"], "dc": dc, "du": du, "dp": dp, "df_pp": df, "dcos": dct,
            "params": np.array([g["mobility"], g["sigma"], g["lambda_"], g["k_n"], g["sigma_attach"]])}


def _calls(s):
    sim, x, p = s["sim"], s["x"], s["p"]
    keys, ids, offsets = sim.cells_build(p)
    f, _ = sim.f_pp(p, 50)
    return {"r2c": sim.fft_r2c(x), "c2r": sim.fft_c2r(s["X"]), "grad": sim.grad(x), "interpolate": sim.interpolate(x, p),
            "spread": sim.spread(p, s["f"]), "f_pp": f, "keys": keys, "ids": ids, "offsets": offsets}


def work(case):
    """Per step: 44 full-grid field passes (every 3-D transform reads its
    input and writes its output once, everything element-wise fused into
    them) and 13 real transforms of 2.5 V log2 V operations; a reversed step
    has 17 transforms more and the recomputed step's 13.  Reading a field
    costs its transform and one write."""
    V = float(case["nx"] * case["ny"] * case["nz"])
    b = 4.0 if case["precision"] == "mixed" else 8.0
    fft = 2.5 * V * math.log2(V)
    part = 500.0 * case["n_p"]
    if case["kind"] == "calls":
        return {"bytes": 8.0 * 11 * V + part, "flops": 6 * fft}
    n = case["steps"]
    if case["kind"] == "gradient":
        return {"bytes": n * (44.0 + 44.0 + 58.0) * V * b + 12.0 * 8 * V + n * 3 * part, "flops": n * 43.0 * fft}
    return {"bytes": n * (44.0 * V * b + part) + 11.0 * V * b, "flops": (13.0 * n + 3.0) * fft}


# ------------------------------------------------------- the same in 64 bits


class _Exact:
    """The reference's iteration in plain torch, 64 bits, full complex
    transforms (x fastest, arrays [z][y][x])."""

    def __init__(self, case, device):
        P = _params(case)
        self.P, self.dev = P, device
        self.shape = (P.nz, P.ny, P.nx)
        self.N = torch.tensor([P.nx, P.ny, P.nz], device=device)
        self.L = torch.tensor([P.lx, P.ly, P.lz], dtype=torch.float64, device=device)

        def waves(n, length):
            q = torch.arange(n, device=device, dtype=torch.float64)
            return torch.where(q <= n // 2, q, q - n) * 2.0 * REF_PI / length  # +N/2 at the Nyquist index

        self.k = [waves(P.nx, P.lx).view(1, 1, -1), waves(P.ny, P.ly).view(1, -1, 1), waves(P.nz, P.lz).view(-1, 1, 1)]
        self.kg = []  # the gradient's, Nyquist index zeroed
        for a, n in enumerate((P.nx, P.ny, P.nz)):
            k = self.k[a].clone()
            k.view(-1)[n // 2] = 0.0
            self.kg.append(k)
        self.k2 = self.k[0] ** 2 + self.k[1] ** 2 + self.k[2] ** 2
        z = lambda v: torch.tensor(v, dtype=torch.float64, device=device)  # noqa: E731
        self.lam, self.M, self.kn, self.sig = z(P.lambda_), z(P.mobility), z(P.k_n), z(P.sigma)
        self.conserve, self.couple = case["conserve"], case["couple"]
        self.t = 0
        self.hist = None

    def fft(self, a):
        return torch.fft.fftn(a)

    def back(self, a):
        return torch.fft.ifftn(a).real

    def bulk(self, c):
        return (c * c * c - c) * (self.lam / self.P.epsilon ** 2)

    def grad(self, ch):
        return [self.back(1j * k * ch) for k in self.kg]

    def nodes(self, p):
        h = self.L / self.N
        q = p / h
        i = torch.floor(q)
        w = q - i
        i = i.long() % self.N
        return i, (i + 1) % self.N, w

    def corners(self, p):
        i0, i1, w = self.nodes(p)
        for a in (0, 1):
            for b in (0, 1):
                for c in (0, 1):
                    ix, iy, iz = (i1 if a else i0)[:, 0], (i1 if b else i0)[:, 1], (i1 if c else i0)[:, 2]
                    wt = (w[:, 0] if a else 1 - w[:, 0]) * (w[:, 1] if b else 1 - w[:, 1]) * (w[:, 2] if c else 1 - w[:, 2])
                    yield (iz * self.P.ny + iy) * self.P.nx + ix, wt

    def at(self, f, p):
        return sum(f.reshape(-1)[node] * wt for node, wt in self.corners(p))

    def spread(self, p, f):
        P = self.P
        dv = P.lx * P.ly * P.lz / (P.nx * P.ny * P.nz)
        out = [torch.zeros(P.nx * P.ny * P.nz, dtype=torch.float64, device=self.dev) for _ in range(3)]
        for node, wt in self.corners(p):
            out = [o.index_add(0, node, f[:, a] / dv * wt) for a, o in enumerate(out)]
        return [o.view(self.shape) for o in out]

    def cells(self, p):
        P = self.P
        nc = [int(math.floor(length / P.r_c)) for length in (P.lx, P.ly, P.lz)]
        dc = [math.fmod(length, P.r_c) / n + P.r_c for length, n in zip((P.lx, P.ly, P.lz), nc)]
        at = torch.floor(p / torch.tensor(dc, dtype=torch.float64, device=self.dev)).long()
        key = at[:, 0] + at[:, 1] * nc[0] + at[:, 2] * nc[0] * nc[1]
        ids = torch.argsort(key, stable=True)
        count = torch.bincount(key, minlength=nc[0] * nc[1] * nc[2])
        return nc, at, key, ids, torch.cat([count.new_zeros(1), count.cumsum(0)])

    def contacts(self, p, t):
        """k_n ramp (r_eq - |d|) d / |d| over every pair within r_eq."""
        P, n = self.P, p.shape[0]
        with torch.no_grad():
            nc, at, _, ids, off = self.cells(p)
            me = torch.arange(n, device=self.dev)
            ii, jj = [], []
            for dz in (-1, 0, 1):
                for dy in (-1, 0, 1):
                    for dx in (-1, 0, 1):
                        cell = (at[:, 0] + dx) % nc[0] + ((at[:, 1] + dy) % nc[1]) * nc[0] \
                            + ((at[:, 2] + dz) % nc[2]) * nc[0] * nc[1]
                        m = off[cell + 1] - off[cell]
                        i = torch.repeat_interleave(me, m)
                        first = torch.repeat_interleave(m.cumsum(0) - m, m)
                        j = ids[torch.repeat_interleave(off[cell], m) + torch.arange(i.numel(), device=self.dev) - first]
                        d = p[i] - p[j]
                        d = d - self.L * torch.round(d / self.L)
                        keep = (i != j) & ((d * d).sum(1) < P.r_eq ** 2)
                        ii.append(i[keep])
                        jj.append(j[keep])
            i, j = torch.cat(ii), torch.cat(jj)
        thr = 0.2 * P.t_end
        ramp = t / thr if t < thr else 1.0
        d = p[i] - p[j]
        d = d - self.L * torch.round(d / self.L).detach()
        dn = torch.sqrt((d * d).sum(1, keepdim=True))
        return torch.zeros_like(p).index_add(0, i, (P.r_eq - dn) * ramp * self.kn * d / dn)

    def attach(self, phi, g, r, ct):
        P = self.P
        gn = torch.sqrt((g * g).sum(1))
        on = (phi.abs() <= math.tanh(2.0)) & (gn != 0)
        ph = torch.where(on, phi, torch.zeros_like(phi))
        d = 0.5 * torch.log((1 + ph) / (1 - ph)) * math.sqrt(2.0) * P.epsilon
        mag = -P.A * P.pi * (d - r * ct) * self.sig
        on = on & (d.abs() < r)
        gs = torch.where(on, gn, torch.ones_like(gn))
        return torch.where(on[:, None], g / gs[:, None] * mag[:, None], torch.zeros_like(g))

    def wrap(self, p):
        q = p + self.L
        return q - self.L * torch.floor(q / self.L).detach()

    def start(self, c, u, p, r, ct, f):
        self.c, self.u = c.view(self.shape), u
        self.p, self.r, self.ct, self.fpp = p, r, ct, f
        self.fpi = torch.zeros_like(p)

    def step(self):
        P, dt, M, lam = self.P, self.P.dt, self.M, self.lam
        c = self.c
        ch, fh = self.fft(c), self.fft(self.bulk(c))
        g = self.grad(ch)
        conv = self.fft(sum(a * b for a, b in zip(self.u, g)))
        if self.conserve:
            conv = torch.where(self.k2 == 0, torch.zeros_like(conv), conv)
        k2, k4 = self.k2, self.k2 ** 2
        if self.t == 0:
            new = (ch - k2 * (dt * M) * fh - conv * dt) / (k4 * (dt * M * lam) + 1)
        else:
            co, fo, Co = self.hist
            new = (4 * ch - co - k2 * (4 * dt * M) * fh + k2 * (2 * dt * M) * fo - conv * (4 * dt) + Co * (2 * dt)) \
                / (k4 * (2 * dt * M * lam) + 3)
        self.hist = (ch, fh, conv)
        del ch, fh, conv, g
        c = self.c = self.back(new)
        mu = self.back(lam * k2 * new + self.fft(self.bulk(c)))
        g = self.grad(new)
        del new
        force = [mu * a for a in g]
        del mu
        if P.n_p:
            force = [a + b for a, b in zip(force, self.spread(self.p, self.fpp))]
        force[2] = force[2] + ((c + 1) / 2 * P.rho1 + (1 - c) / 2 * P.rho2) * P.gravity
        fh = [self.fft(a) for a in force]
        del force
        ks = torch.where(k2 == 0, torch.ones_like(k2), k2)
        dot = sum(k * a for k, a in zip(self.k, fh)) / ks
        self.u = [self.back(torch.where(k2 == 0, torch.zeros_like(a), (a - k * dot) / (ks * P.mu))) for k, a in zip(self.k, fh)]
        del fh, dot, ks
        if P.n_p:
            self.particles(g)
        self.t += 1

    def particles(self, g):
        P = self.P
        old = p = self.p
        v0 = None
        for _ in range(2):  # Heun: p1 = p + v dt, then p + (v + v(p1)) dt / 2
            phi = self.at(self.c, p)
            dphi = torch.stack([self.at(a, p) for a in g], dim=1)
            self.fpi = self.attach(phi, dphi, self.r, self.ct)
            self.fpp = self.contacts(p, self.t + 1)
            v = (self.fpi + self.fpp) / (6 * P.pi * P.mu * self.r[:, None])
            if self.couple:
                v = v + torch.stack([self.at(a, p) for a in self.u], dim=1)
            p = self.wrap(old + v * P.dt if v0 is None else old + (v0 + v) * (0.5 * P.dt))
            v0 = v
        self.p = p


def exact(case, seed):
    dev = _device()
    P = _params(case)
    E = _Exact(case, dev)
    c = _phase(case, seed, dev)
    p, r, ct, f = (torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in _particles(case, seed))
    V, n = P.nx * P.ny * P.nz, P.n_p
    if case["kind"] == "calls":
        x = c.view(E.shape)
        X = torch.fft.rfftn(x).transpose(1, 2).reshape(-1)
        _, _, key, ids, off = E.cells(p)
        g = torch.stack(E.grad(E.fft(x))).reshape(-1)
        got = {"r2c": X, "c2r": x.reshape(-1), "grad": g, "interpolate": E.at(x, p).view(n, 1),
               "spread": torch.stack(E.spread(p, f)).reshape(-1), "f_pp": E.contacts(p, 50.0).reshape(-1),
               "keys": key.int(), "ids": ids.int(), "offsets": off.int()}
        return {k: v.cpu().numpy() for k, v in got.items()}
    if case["kind"] != "gradient":
        with torch.no_grad():
            E.start(c, [torch.zeros(E.shape, dtype=torch.float64, device=dev) for _ in range(3)], p, r, ct, f)
            for _ in range(case["steps"]):
                E.step()
            out = {"phase": E.c.reshape(-1), "velocity": torch.cat([a.reshape(-1) for a in E.u])}
            if n:
                out.update(positions=E.p.reshape(-1), f_pp=E.fpp.reshape(-1), f_pi=E.fpi.reshape(-1))
            return out
    u = 0.01 * _normals(3 * V, seed, 3, dev)
    leaves = [c, u, p, f, ct, E.M, E.lam, E.kn, E.sig]
    for a in leaves:
        a.requires_grad_(True)
    E.start(c, [u[a * V:(a + 1) * V].view(E.shape) for a in range(3)], p, r, ct, f)
    for _ in range(case["steps"]):
        E.step()
    rng = np.random.default_rng(1000 * seed + 6)
    put = lambda a: torch.from_numpy(a).to(dev)  # noqa: E731
    dp, df = put(rng.standard_normal(3 * n)), put(rng.standard_normal(3 * n))
    loss = (E.c.reshape(-1) * _normals(V, seed, 4, dev)).sum()
    loss = loss + (torch.cat([a.reshape(-1) for a in E.u]) * _normals(3 * V, seed, 5, dev)).sum()
    loss = loss + (E.p.reshape(-1) * dp).sum() + (E.fpp.reshape(-1) * df).sum()
    dc, du, dq, dfp, dct, dM, dl, dk, ds = torch.autograd.grad(loss, leaves)
    total = ds + 3.0 * P.epsilon / (2.0 * math.sqrt(2.0)) * dl + 0.5 * dk  # lambda and k_n follow sigma
    return {"phase": E.c.detach().reshape(-1), "dc": dc.reshape(-1), "du": du.reshape(-1), "dp": dq.reshape(-1),
            "df_pp": dfp.reshape(-1), "dcos": dct, "params": torch.stack([dM, total, dl, dk, ds])}
