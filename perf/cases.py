"""Performance cases: the work that a user of this framework has it do.

A case is one call cycle through the public Python entry points (`abi.System`,
`abi.Batch`): the state goes in from pinned host memory, a number of steps runs
on the device, and the resulting state comes back, as a caller of the C-ABI
does it (a `DoStep` of the drop-in, a served request, a bench step).  The
kinds are

* ``system``: one particle system of the Chimera, vortex or vortex-arrays model,
* ``batch``: many systems of uneven N, resident in one batch,
* ``order``: the global and local order parameters of one system, which
  observers record of every frame.

`exact` restates the models in 64 bits with plain torch.
"""
import math

import numpy as np
import torch

from spc2_langevin_integration_gb300 import abi

STEPPERS = {"euler": abi.STEPPER_EULER, "srk": abi.STEPPER_SRK, "rk4": abi.STEPPER_RK4}
PRECISIONS = {"fp64": abi.PRECISION_FP64, "fp32c": abi.PRECISION_FP32C, "fp32x": abi.PRECISION_FP32X}
MODELS = {"chimera": abi.MODEL_CHIMERA, "vortex": abi.MODEL_VORTEX, "vortex_arrays": abi.MODEL_VORTEX_ARRAYS}

# the parameter sets of the repository's own workloads, by the name a case gives
PARAMS = {
    # the unit-box Chimera system and the large deterministic one (D = 0)
    "chimera": dict(v0=0.01, sigma=1.0, alpha=1.45, D_phi=0.005),
    "chimera_d0": dict(v0=0.01, sigma=1.0, alpha=1.45, D_phi=0.0),
    # the vortex system: natural frequencies N(0, 0.5^2), no phase lag
    "vortex": dict(v0=0.02, sigma=2.0, alpha=0.0, D_phi=0.01),
    # the reference's vortex-array parameters
    "vortex_arrays": dict(velocity=0.1, mu_plus=100.0, mu_minus=100.0, xi_a=0.04, xi_r=0.02, D_phi=0.01,
                          kappa=20.0),
}


def _system(name, model, params, stepper, precision, n, density, rho, dt, steps, graph, neighbour="cell",
            state="uniform", units=False):
    return dict(name=name, kind="system", model=model, params=params, stepper=stepper, precision=precision,
                n=n, density=density, rho=rho, dt=dt, steps=steps, graph=graph, neighbour=neighbour,
                state=state, units=units)


def _batch(name, precision, systems, n_lo, n_hi, vortex, steps):
    return dict(name=name, kind="batch", precision=precision, systems=systems, n_lo=n_lo, n_hi=n_hi,
                vortex=vortex, steps=steps, dt=0.01)


def listed():
    return [
        # one DoStep of the drop-in on the unit-box Chimera system: state in, one
        # step, state out; launches and latency count
        _system("chimera_dostep_fp64", "chimera", "chimera", "euler", "fp64", 1024, 1024.0, 0.1, 0.01, 1, False),
        # the same system advanced by a 100-step graph between observed frames
        _system("chimera_run100_fp64", "chimera", "chimera", "euler", "fp64", 1024, 1024.0, 0.1, 0.01, 100, True),
        # a small box with rho > L / 4: the reference's all-pairs form
        _system("chimera_allpairs_fp64", "chimera", "chimera", "euler", "fp64", 2000, 2000.0, 0.3, 0.01, 10, True),
        # the vortex system of the headline, plain FP64: the drop-in's default
        # cell list, and Verlet rows
        _system("vortex_srk_fp64_cell", "vortex", "vortex", "srk", "fp64", 65536, 1024.0, 0.25, 0.005, 10, True),
        _system("vortex_srk_fp64_verlet", "vortex", "vortex", "srk", "fp64", 65536, 1024.0, 0.25, 0.005, 10, True,
                neighbour="verlet"),
        # the same in FP32C from the initial state, and in FP32X from a clustered
        # state with cell units on, as the tuner leaves it there
        _system("vortex_srk_fp32c", "vortex", "vortex", "srk", "fp32c", 65536, 1024.0, 0.25, 0.005, 20, True),
        _system("vortex_srk_fp32x_clustered", "vortex", "vortex", "srk", "fp32x", 65536, 1024.0, 0.25, 0.005, 20,
                True, state="clustered", units=True),
        # the large deterministic Chimera system, RK4 in FP32C
        _system("chimera_rk4_fp32c_large", "chimera", "chimera_d0", "rk4", "fp32c", 1 << 22, 1024.0, 0.25, 0.01, 2,
                True),
        # a parameter sweep: many Chimera systems of uneven N in one batch, FP32X
        # (the form that keeps the ensemble's order parameters)
        _batch("ensemble_euler_fp32x", "fp32x", 96, 256, 32768, False, 50),
        # systems of a served request stream, Chimera and vortex mixed, FP32C
        _batch("served_euler_fp32c", "fp32c", 24, 512, 262144, True, 10),
        # the reference's second model
        _system("vortex_arrays_srk_fp64", "vortex_arrays", "vortex_arrays", "srk", "fp64", 12800, 800.0, 0.2, 0.01,
                2, True),
        # an observer's summary of a frame
        dict(name="order_parameters", kind="order", n=65536, density=1024.0, rho=0.25),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["small", "allpairs", "fp64", "float", "float", "rk4", "batch", "batch", "arrays", "order"])
    if kind == "small":
        n = _log(rng, 300, 6000)
        steps = rng.choice([1, 100])
        c = _system("", "chimera", "chimera", "euler", rng.choice(["fp64", "fp64", "fp32x", "fp32c"]), n, 1000.0,
                    rng.uniform(0.05, 0.12), 0.01, steps, steps > 1)
        if c["precision"] == "fp32c":
            c["steps"] = min(steps, 10)
    elif kind == "allpairs":
        n = _log(rng, 100, 2500)
        c = _system("", "chimera", "chimera", rng.choice(["euler", "srk"]), "fp64", n, float(n),
                    rng.uniform(0.26, 0.45), 0.01, 5, True)
    elif kind == "fp64":
        n = _log(rng, 4000, 120000)
        c = _system("", "vortex", "vortex", "srk", "fp64", n, rng.uniform(400.0, 1100.0), rng.uniform(0.2, 0.26),
                    0.005, rng.choice([2, 5, 10]), True, neighbour=rng.choice(["cell", "verlet"]),
                    state=rng.choice(["uniform", "uniform", "clustered"]))
    elif kind == "float":
        n = _log(rng, 8000, 400000)
        state = rng.choice(["uniform", "clustered"])
        c = _system("", "vortex", "vortex", "srk", rng.choice(["fp32c", "fp32x"]), n, rng.uniform(400.0, 1100.0),
                    rng.uniform(0.2, 0.26), 0.005, rng.choice([5, 10, 20]), True, state=state,
                    units=state == "clustered")
    elif kind == "rk4":
        n = _log(rng, 20000, 3000000)
        c = _system("", "chimera", "chimera_d0", "rk4", rng.choice(["fp32c", "fp32x"]), n, 1024.0,
                    rng.uniform(0.15, 0.25), 0.01, 1, True)
    elif kind == "batch":
        served = rng.random() < 0.5
        c = _batch("", rng.choice(["fp32x", "fp32c", "fp64"]), rng.randint(2, 24) if served else rng.randint(8, 96),
                   512 if served else 256, 200000 if served else 32768, served, rng.choice([5, 10]))
    elif kind == "arrays":
        n = _log(rng, 2000, 26000)
        c = _system("", "vortex_arrays", "vortex_arrays", "srk", "fp64", n, rng.uniform(400.0, 1000.0),
                    rng.uniform(0.1, 0.2), 0.01, 2, True)
    else:
        c = dict(kind="order", n=_log(rng, 1000, 262144), density=rng.uniform(300.0, 1100.0),
                 rho=rng.uniform(0.1, 0.25))
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# Inputs
def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def _uniform(rng, n, L):
    st = _pinned(3 * n)
    st[0::3] = rng.uniform(0.0, L, n)
    st[1::3] = rng.uniform(0.0, L, n)
    st[2::3] = rng.uniform(-np.pi, np.pi, n)
    return st


def _clustered(rng, n, L, rho):
    """Half of the particles in clusters about a cutoff wide, with phases
    aligned inside a cluster, over a uniform rest: cells of a few to several
    hundred particles, as the vortex system leaves them after some thousand
    steps."""
    st = _uniform(rng, n, L)
    m = max(2, n // 800)
    k = rng.choice(m, n, p=rng.dirichlet(np.ones(m)))
    centre, phase = rng.uniform(0.0, L, (m, 2)), rng.uniform(-np.pi, np.pi, m)
    inside = rng.random(n) < 0.5
    for d in (0, 1):
        x = centre[k, d] + rng.normal(0.0, rho, n)
        x -= np.floor(x / L) * L
        st[d::3] = np.where(inside & (x < L), x, st[d::3])
    st[2::3] = np.where(inside, phase[k] + rng.normal(0.0, 0.4, n), st[2::3])
    return st


def _box(case):
    return math.sqrt(case["n"] / case["density"])


def _make_system(case, seed):
    """(n, abi.Params, state, omega or None) of a system or order case."""
    rng = np.random.default_rng(seed)
    n, L = case["n"], _box(case)
    if case["kind"] == "order":
        p = abi.make_params(L=L, rho=case["rho"], stepper=abi.STEPPER_SRK, seed=seed, **PARAMS["chimera"])
        return n, p, _uniform(rng, n, L), None
    prm = dict(PARAMS[case["params"]], rho=case["rho"])
    if case["model"] == "vortex_arrays":
        p = abi.make_va_params(L=L, stepper=STEPPERS[case["stepper"]], seed=seed, **prm)
    else:
        verlet = case["neighbour"] == "verlet"
        p = abi.make_params(L=L, model=MODELS[case["model"]], stepper=STEPPERS[case["stepper"]],
                            precision=PRECISIONS[case["precision"]], skin=0.05, seed=seed,
                            neighbour=abi.NEIGHBOUR_VERLET if verlet else abi.NEIGHBOUR_CELL, **prm)
    st = _clustered(rng, n, L, case["rho"]) if case["state"] == "clustered" else _uniform(rng, n, L)
    return n, p, st, rng.normal(0.0, 0.5, n) if case["model"] == "vortex" else None


def _make_batch(case, seed):
    """[(n, abi.Params, state, omega or None)] of a batch case.  The systems'
    sizes are the case's own (evenly spread over the logarithm), so that every
    seed asks for the same work; parameters and states are the seed's."""
    rng = np.random.default_rng(seed)
    out = []
    for k in range(case["systems"]):
        n = int(round(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** ((k + 0.5) / case["systems"])))
        vortex = case["vortex"] and k % 2 == 1
        p = abi.make_params(L=math.sqrt(n / 1000.0), v0=0.01, sigma=rng.uniform(0.5, 2.0),
                            rho=0.05 + 0.1 * ((k * 0.6180339887498949) % 1.0),
                            alpha=0.0 if vortex else rng.uniform(1.2, 1.6), D_phi=rng.uniform(0.0, 0.02),
                            model=abi.MODEL_VORTEX if vortex else abi.MODEL_CHIMERA, stepper=abi.STEPPER_EULER,
                            precision=PRECISIONS[case["precision"]], seed=seed, system_id=k)
        out.append((n, p, _uniform(rng, n, p.L), rng.normal(0.0, 0.5, n) if vortex else None))
    return out


def prepare(case, seed):
    if case["kind"] == "batch":
        systems = _make_batch(case, seed)
        b = abi.Batch(abi.STEPPER_EULER, PRECISIONS[case["precision"]], len(systems), sum(s[0] for s in systems),
                      sum(abi.cells_of(s[1].L, s[1].rho) for s in systems))
        slots = [b.admit(n, p, st, om) for n, p, st, om in systems]
        out = _pinned(3 * sum(s[0] for s in systems))
        views = np.split(out, np.cumsum([3 * s[0] for s in systems])[:-1])
        return dict(case=case, batch=b, slots=slots, out=out, views=views)
    n, p, st, om = _make_system(case, seed)
    s = abi.System(n, p)
    s.upload_state(st)
    if om is not None:
        s.upload_omega(om)
    if case["kind"] == "order":
        return dict(case=case, system=s, state=st)
    if case["units"]:
        s.set_tuning(abi.TUNE_CELL_UNITS, 1)
    if case["graph"]:
        s.prepare_graph(case["dt"], case["steps"])
    return dict(case=case, system=s, state=st, out=_pinned(3 * n))


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.step(case["dt"], case["steps"], graph=True)
        for slot, view in zip(state["slots"], state["views"]):
            b.download(slot, view)
        return state["out"]
    s = state["system"]
    s.upload_state(state["state"])
    if case["kind"] == "order":
        return s.order_params()
    s.step(case["dt"], case["steps"], graph=case["graph"])
    return s.download_state(state["out"])


# ---------------------------------------------------------------------------
# What a pass cannot do without
def _neighbours(n, L, rho):
    return n * math.pi * rho * rho * n / (L * L)


def work(case):
    if case["kind"] == "batch":
        systems = [(s[0], s[1].L, s[1].rho, 32 if s[3] is not None else 24) for s in _make_batch(case, 0)]
        evals, steps = 1, case["steps"]
    else:
        systems = [(case["n"], _box(case), case["rho"], 32 if case.get("model") == "vortex" else 24)]
        evals = {"euler": 1, "srk": 2, "rk4": 4}[case.get("stepper", "euler")]
        steps = case.get("steps", 1)
    # the state (and frequencies) in, the state out; per neighbour pair and
    # evaluation the distance (5), the test (1) and the two sums (2, with a
    # weight 4)
    out_bytes = 0 if case["kind"] == "order" else 24
    return {"bytes": float(sum(n * (b + out_bytes) for n, _, _, b in systems)),
            "flops": float(sum(10.0 * _neighbours(n, L, rho) for n, L, rho, _ in systems) * evals * steps)}


# ---------------------------------------------------------------------------
# The models in 64 bits
class _Philox:
    """Philox4x32-10 (Salmon et al., SC'11) normals of (seed, system, step,
    particle): Box-Muller on two 53-bit uniforms."""

    def __init__(self, seed, ids, local):
        self.seed, self.ids, self.local = seed, ids, local

    def normals(self, step):
        m32 = 0xFFFFFFFF
        c = [self.local.clone(), self.ids.clone(), torch.full_like(self.ids, step & m32),
             torch.full_like(self.ids, step >> 32)]
        k0, k1 = self.seed & m32, (self.seed >> 32) & m32
        for _ in range(10):
            p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57  # modulo 2^64: the bits of the unsigned product
            c = [((p1 >> 32) & m32) ^ c[1] ^ k0, p1 & m32, ((p0 >> 32) & m32) ^ c[3] ^ k1, p0 & m32]
            k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
        u1 = (((c[0] << 21) | (c[1] >> 11)) + 1).double() * 2.0 ** -53
        u2 = ((c[2] << 21) | (c[3] >> 11)).double() * 2.0 ** -53
        r = torch.sqrt(-2.0 * torch.log(u1))
        return r * torch.cos(2.0 * math.pi * u2), r * torch.sin(2.0 * math.pi * u2)


class _Exact:
    """Systems as one set of particles with per-particle constants."""

    def __init__(self, systems, seed):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.dev = dev
        par = lambda f: torch.cat([torch.full((n,), float(f(p)), dtype=torch.float64, device=dev)  # noqa: E731
                                   for n, p, _, _ in systems])
        state = torch.from_numpy(np.concatenate([st for _, _, st, _ in systems])).to(dev).view(-1, 3)
        self.x, self.y, self.phi = (state[:, d].clone() for d in range(3))
        self.omega = torch.cat([torch.zeros(n, dtype=torch.float64) if om is None else torch.from_numpy(om)
                                for n, _, _, om in systems]).to(dev)
        self.L, self.v0, self.sigma, self.alpha, self.D = (par(lambda p, k=k: getattr(p, k))
                                                           for k in ("L", "v0", "sigma", "alpha", "D_phi"))
        self.sizes = [n for n, _, _, _ in systems]
        self.p0 = systems[0][1]
        ids = torch.cat([torch.full((n,), p.system_id, dtype=torch.int64, device=dev) for n, p, _, _ in systems])
        local = torch.cat([torch.arange(n, dtype=torch.int64, device=dev) for n in self.sizes])
        self.noise = _Philox(seed, ids, local)
        # cells of side L / int(L / rho), or one cell for rho > L / 4
        nc = [int(p.L / p.rho) if p.rho <= 0.25 * p.L else 1 for _, p, _, _ in systems]
        c0 = np.concatenate([[0], np.cumsum([k * k for k in nc])])
        self.ncell = int(c0[-1])
        self.nc = torch.cat([torch.full((n,), k, dtype=torch.int64, device=dev) for n, k in zip(self.sizes, nc)])
        self.c0 = torch.cat([torch.full((n,), int(c), dtype=torch.int64, device=dev) for n, c in zip(self.sizes, c0)])
        nbr, cl, cr = [], [], []
        for k, c, (_, p, _, _) in zip(nc, c0, systems):
            i = torch.arange(k * k, device=dev)
            cx, cy = i % k, i // k
            nbr.append(torch.stack([int(c) + (cy + oy) % k * k + (cx + ox) % k for oy in (-1, 0, 1) for ox in (-1, 0, 1)]
                                   if k > 1 else [i * 0 + int(c)] + [i * 0 - 1] * 8, 1))
            cl.append(torch.full((k * k,), p.L, dtype=torch.float64, device=dev))
            cr.append(torch.full((k * k,), p.rho, dtype=torch.float64, device=dev))
        self.nbr, self.cell_L, self.cell_rho = torch.cat(nbr), torch.cat(cl), torch.cat(cr)

    def wrap(self, x, y):
        out = (x < 0) | (x >= self.L) | (y < 0) | (y >= self.L)
        return (torch.where(out, x - torch.floor(x / self.L) * self.L, x),
                torch.where(out, y - torch.floor(y / self.L) * self.L, y))

    def cells(self, x, y):
        """Members of every cell, [ncell, capacity], -1 where there is none."""
        cx, cy = ((v / self.L * self.nc).long().clamp(min=0) for v in (x, y))
        cell = self.c0 + torch.minimum(cy, self.nc - 1) * self.nc + torch.minimum(cx, self.nc - 1)
        order = torch.argsort(cell, stable=True)
        count = torch.bincount(cell, minlength=self.ncell)
        start = torch.cumsum(count, 0) - count
        table = torch.full((self.ncell, int(count.max())), -1, dtype=torch.int64, device=self.dev)
        sc = cell[order]
        table[sc, torch.arange(len(order), device=self.dev) - start[sc]] = order
        return table

    def pairs(self, x, y):
        """(i, j, dx, dy, within) of neighbouring cells, in pieces: i [c, a, 1], j [c, 1, b]."""
        table = self.cells(x, y)
        cap = table.shape[1]
        filled = torch.nonzero(table[:, 0] >= 0)[:, 0]
        piece = max(1, int(4e7) // (cap * cap))
        for a in range(0, len(filled), piece):
            c = filled[a:a + piece]
            i = table[c][:, :, None]
            L, rho = self.cell_L[c][:, None, None], self.cell_rho[c][:, None, None]
            for q in range(9):
                cj = self.nbr[c, q]
                if bool((cj < 0).all()):
                    continue
                j = torch.where((cj < 0)[:, None], -1, table[cj.clamp(min=0)])[:, None, :]
                dx, dy = x[j] - x[i], y[j] - y[i]
                dx, dy = (d - torch.trunc(d * 2.0 / L) * L for d in (dx, dy))
                within = (dx * dx + dy * dy <= rho * rho) & (i >= 0) & (j >= 0) & (i != j)
                yield i, j, dx, dy, within

    def sums(self, x, y, columns):
        """Neighbour count and, for every column of values, its sum over the neighbours."""
        n = len(x)
        v = torch.cat([torch.stack(columns, 1), torch.ones(n, 1, dtype=torch.float64, device=self.dev)], 1)
        out = torch.zeros(n + 1, v.shape[1], dtype=torch.float64, device=self.dev)
        for i, j, _, _, within in self.pairs(x, y):
            s = torch.bmm(within.double(), v[j[:, 0, :]])
            out.index_add_(0, torch.where(i < 0, n, i).reshape(-1), s.reshape(-1, v.shape[1]))
        return out[:n, -1], [out[:n, k] for k in range(len(columns))]

    def rate(self, x, y, phi):
        """Alignment rate (0 when isolated), n_i and sum_j cos(phi_j - phi_i - alpha)."""
        n, (sc, ss) = self.sums(x, y, [torch.cos(phi), torch.sin(phi)])
        ct, st = torch.cos(phi + self.alpha), torch.sin(phi + self.alpha)
        return torch.where(n > 0, self.sigma * (ss * ct - sc * st) / n.clamp(min=1), 0.0), n, sc * ct + ss * st

    def srk_update(self, rate, a0, a1, dt, step):
        d0, d1 = self.v0 * torch.cos(self.phi), self.v0 * torch.sin(self.phi)
        u1, u2 = self.noise.normals(step)
        s2d, sdt = torch.sqrt(2.0 * self.D), math.sqrt(dt)
        dw, dz = u1 * sdt, 0.5 * dt * sdt * (u1 + u2 / math.sqrt(3.0))
        x = self.x + (d0 * dt - s2d * d1 * dz - 0.5 * (rate * d1 + self.D * d0) * dt * dt)
        y = self.y + (d1 * dt + s2d * d0 * dz + 0.5 * (rate * d0 - self.D * d1) * dt * dt)
        self.phi = self.phi + ((self.omega + rate) * dt + s2d * dw + a0 * dz + 0.5 * a1 * dt * dt)
        self.x, self.y = (v - torch.floor(v / self.L) * self.L for v in (x, y))

    def step_euler(self, dt, step):
        x, y = self.wrap(self.x, self.y)
        rate, _, _ = self.rate(x, y, self.phi)
        z, _ = self.noise.normals(step)
        x, y = self.x + dt * self.v0 * torch.cos(self.phi), self.y + dt * self.v0 * torch.sin(self.phi)
        self.phi = self.phi + (dt * (self.omega + rate) + math.sqrt(dt) * torch.sqrt(2.0 * self.D) * z)
        self.x, self.y = (v - torch.floor(v / self.L) * self.L for v in (x, y))

    def step_srk(self, dt, step):
        if self.p0.model == abi.MODEL_VORTEX_ARRAYS:
            return self.srk_update(*self.arrays_rates(), dt, step)
        x, y = self.wrap(self.x, self.y)
        rate, n, scos = self.rate(x, y, self.phi)
        c, s = torch.cos(self.phi), torch.sin(self.phi)
        _, (dc, ds) = self.sums(x, y, [rate * c, rate * s])
        ct, st = torch.cos(self.phi + self.alpha), torch.sin(self.phi + self.alpha)
        m = n.clamp(min=1)
        a0 = scos / m * -torch.sqrt(2.0 * self.D)
        a1 = (dc * ct + ds * st - rate * scos) / m - 2.0 * self.D * rate
        return self.srk_update(rate, a0, a1, dt, step)

    def step_rk4(self, dt, step):
        k = [[torch.zeros_like(self.x) for _ in range(3)] for _ in range(4)] if step == 0 else self.k
        self.k = k
        for s, (coef, prev) in enumerate(((0.0, 0), (0.5, 0), (0.5, 1), (1.0, 2))):
            x, y, phi = (v + coef * dt * d for v, d in zip((self.x, self.y, self.phi), k[prev]))
            x, y = self.wrap(x, y)
            rate, n, _ = self.rate(x, y, phi)
            k[s] = [self.v0 * torch.cos(phi), self.v0 * torch.sin(phi), torch.where(n > 0, rate, k[s][2])]
        dx, dy, dp = (k[0][d] + 2.0 * k[1][d] + 2.0 * k[2][d] + k[3][d] for d in range(3))
        x, y = self.x + dx * dt / 6.0, self.y + dy * dt / 6.0
        self.phi = self.phi + dp / 6.0 * dt
        self.x, self.y = (v - torch.floor(v / self.L) * self.L for v in (x, y))

    def arrays_rates(self):
        """Vortex arrays: phase rate and the SRK form's two additional terms."""
        p, n = self.p0, len(self.x)
        x, y = self.wrap(self.x, self.y)
        phi = self.phi
        vx, vy = self.v0 * torch.cos(phi), self.v0 * torch.sin(phi)
        w = p.rho - p.xi_a

        def total(terms):
            out = torch.zeros(n + 1, dtype=torch.float64, device=self.dev)
            return out, lambda i, t: out.index_add_(0, torch.where(i < 0, n, i).reshape(-1), t.sum(2).reshape(-1))

        def pair(i, j, dx, dy, within):
            dr = torch.sqrt(dx * dx + dy * dy)
            near = dr < p.xi_a
            inside = dr < p.rho
            f = torch.where(near, p.mu_plus * (1.0 - dr * dr / p.xi_a ** 2),
                            torch.where(inside, -p.mu_minus * 4.0 * (dr - p.xi_a) * (p.rho - dr) / w / w, 0.0))
            g = torch.where(near, p.mu_plus * -2.0 * dr / p.xi_a / p.xi_a,
                            torch.where(inside, -p.mu_minus * 4.0 * (-2.0 * dr + p.rho + p.xi_a) / w / w, 0.0))
            coh = within & (dr <= p.xi_r)
            return torch.where(within, dr, 1.0), f, g, phi[j] - phi[i], torch.atan2(dy, dx) - phi[i], coh

        (al, add_al), (co, add_co), (n1, add_n1), (n2, add_n2) = (total(None) for _ in range(4))
        for i, j, dx, dy, within in self.pairs(x, y):
            dr, f, g, d, th, coh = pair(i, j, dx, dy, within)
            add_al(i, torch.where(within, f * torch.sin(d), 0.0))
            add_co(i, torch.where(coh, -p.kappa * torch.sin(th), 0.0))
            add_n1(i, within.double())
            add_n2(i, coh.double())
        n1, n2 = n1[:n], n2[:n]
        m1, m2 = n1.clamp(min=1), n2.clamp(min=1)
        rate = torch.where(n1 > 0, al[:n] / m1, 0.0) + torch.where(n2 > 0, co[:n] / m2, 0.0)
        (a0, add_a0), (a1, add_a1) = total(None), total(None)
        for i, j, dx, dy, within in self.pairs(x, y):
            dr, f, g, d, th, coh = pair(i, j, dx, dy, within)
            dvx, dvy, dd = vx[j] - vx[i], vy[j] - vy[i], rate[j] - rate[i]
            s, c = torch.sin(d), torch.cos(d)
            add_a0(i, torch.where(within, -f * c / m1[i], 0.0))
            add_a1(i, torch.where(within, ((dvx * g * dx / dr + dvy * g * dy / dr) * s + dd * f * c
                                           - 2.0 * p.D_phi * s * f) / m1[i], 0.0))
            s, c = torch.sin(th), torch.cos(th)
            add_a0(i, torch.where(coh, p.kappa * c / m2[i], 0.0))
            inner = (-dvx * dy + dvy * dx) / dr / dr - rate[i]
            add_a1(i, torch.where(coh, (-p.kappa * inner * c + p.kappa * p.D_phi * s) / m2[i], 0.0))
        return rate, a0[:n] * torch.sqrt(2.0 * self.D), a1[:n]

    def order(self):
        x, y = self.wrap(self.x, self.y)
        c, s = torch.cos(self.phi), torch.sin(self.phi)
        n, (sc, ss) = self.sums(x, y, [c, s])
        re, im = float(c.mean()), float(s.mean())
        local = torch.sqrt((sc + c) ** 2 + (ss + s) ** 2) / (n + 1.0)
        return {"R": math.hypot(re, im), "psi": math.atan2(im, re), "R_local": float(local.mean())}

    def states(self):
        return torch.stack([self.x, self.y, self.phi], 1).cpu().numpy().reshape(-1)


def exact(case, seed):
    if case["kind"] == "batch":
        ref = _Exact(_make_batch(case, seed), seed)
    else:
        ref = _Exact([_make_system(case, seed)], seed)
    if case["kind"] == "order":
        return ref.order()
    step = {"euler": ref.step_euler, "srk": ref.step_srk, "rk4": ref.step_rk4}[case.get("stepper", "euler")]
    for s in range(case["steps"]):
        step(case["dt"], s)
    return ref.states()
