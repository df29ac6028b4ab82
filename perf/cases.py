"""The work a host program has the library do, as timed cases.

A case is one job of such a program: the initial fields go from the host's
own (pinned) arrays to the device, a number of hydro steps run, and the
fields come back, through the package's public entry points
(Solver, BatchSolver, ClosureNet).  The sizes, options and distributions
are those of this repository's control files, tests and benchmark.

``exact`` gives the same results from a plain torch restatement of the
method in FP64 (array expressions over the whole mesh), independent of the
package beyond the initial fields.
"""
import math
import random

import numpy as np
import torch

from bookleaf_f90_gb300 import BatchSolver, Problem, Solver, abi, configs
from bookleaf_f90_gb300.closure import ClosureNet, init_params

MODES = {"fast": abi.FP_FAST, "exact": abi.FP_EXACT, "mixed": abi.FP_MIXED}
LAG_BYTES, EUL_BYTES = 724, 1628      # per zone-cycle, fields read and written once per phase
LAG_FLOPS, EUL_FLOPS = 700, 1400      # per zone-cycle, about, divides and square roots as one


# ------------------------------------------------------------------ cases

def listed():
    return [
        # a host that calls the three entry points itself every step, on the
        # reference's smallest Sod mesh: launches and latency are all of it
        dict(name="sod_100x10_calls", kind="sod", nx=100, ny=10, eul=False, mode="fast",
             drive="calls", steps=40),
        # the benchmark's 400x40 Sod tube in the device time loop
        dict(name="sod_400x40_loop", kind="sod", nx=400, ny=40, eul=False, mode="fast",
             drive="loop", steps=200),
        # the bit-reproducible form, as a validation run uses it
        dict(name="sedov_128_exact_loop", kind="sedov", nx=128, ny=128, eul=False, mode="exact",
             drive="loop", steps=100),
        # an Eulerian (remapped) blast on a mesh of odd size, called per step
        dict(name="sedov_eul_97_calls", kind="sedov", nx=97, ny=97, eul=True, mode="fast",
             drive="calls", steps=50),
        # the headline: Sedov 512x512 with hourglass and sub-zonal control
        dict(name="sedov_512_loop", kind="sedov", nx=512, ny=512, eul=False, mode="fast",
             drive="loop", steps=100),
        # the same mesh as one whole short job: set-up of the context from
        # host arrays, 20 called steps, the fields back
        dict(name="sedov_512_job", kind="sedov", nx=512, ny=512, eul=False, mode="fast",
             drive="job", steps=20),
        # the reference's own Noh form: a polar mesh (no square cells)
        dict(name="noh_polar_300x120_loop", kind="polar", nx=300, ny=120, eul=False, mode="fast",
             drive="loop", steps=150),
        # the demoted form on a ragged Lagrangian mesh
        dict(name="sedov_301_mixed_loop", kind="sedov", nx=301, ny=301, eul=False, mode="mixed",
             drive="loop", steps=100),
        # the largest mesh: Noh 1024x1024 with the remap every step
        dict(name="noh_eul_1024_loop", kind="noh", nx=1024, ny=1024, eul=True, mode="fast",
             drive="loop", steps=32),
        # an ensemble of uneven Eulerian meshes advanced as one batch in the
        # demoted form
        dict(name="ensemble_48_mixed", kind="ensemble", nx=32, ny=256, eul=True, mode="mixed",
             drive="batch", steps=48, meshes=48),
        # two materials, mixed cells under the learned closure
        dict(name="sod2mat_800x80_closure", kind="sod2mat", nx=800, ny=80, tilt=0.2, eul=False,
             mode="fast", drive="loop", steps=100),
        # the closure network's training (forward, backward, Adam)
        dict(name="closure_train_16384", kind="train", samples=16384, batch=256, epochs=2),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sod", "sod", "sedov", "sedov", "noh", "polar", "ensemble", "sod2mat",
                       "train"])
    if kind == "train":
        return dict(kind=kind, samples=_logint(rng, 500, 40000), batch=rng.choice([64, 128, 256, 500]),
                    epochs=rng.randint(1, 3))
    if kind == "ensemble":
        return dict(kind=kind, nx=rng.randint(16, 40), ny=rng.randint(60, 256),
                    eul=rng.random() < 0.7, mode=rng.choice(["fast", "mixed"]), drive="batch",
                    steps=rng.randint(16, 60), meshes=rng.randint(3, 40))
    c = dict(kind=kind, eul=False, mode="fast", drive=rng.choice(["loop", "loop", "calls", "job"]),
             steps=rng.randint(20, 100))
    if kind == "sod":
        c.update(ny=_logint(rng, 3, 70), eul=rng.random() < 0.4)
        c["nx"] = max(8, int(c["ny"] * rng.uniform(5, 15)))
    elif kind == "sedov":
        n = _logint(rng, 20, 520)
        c.update(nx=n, ny=n, eul=rng.random() < 0.3)
    elif kind == "noh":
        n = _logint(rng, 20, 700)
        c.update(nx=n, ny=n, eul=rng.random() < 0.7)
    elif kind == "polar":
        c["nx"] = _logint(rng, 40, 600)
        c["ny"] = max(8, int(c["nx"] * rng.uniform(0.3, 0.5)))
    else:
        c["nx"] = _logint(rng, 100, 1000)
        c.update(ny=max(4, c["nx"] // 10), tilt=rng.uniform(0.1, 0.4))
    if kind != "sod2mat":
        c["mode"] = rng.choice(["fast", "fast", "fast", "mixed", "exact"])
    return c


# ------------------------------------------------------------------ inputs

def _problem(case, seed):
    """One seeded initial state of the case's problem."""
    r = random.Random(seed * 7919 + 13)
    kind, frac = case["kind"], None
    if kind == "sod":
        deck = configs.sod(case["nx"], case["ny"], time_end=1.0e3, eulerian=case["eul"],
                           gamma=r.uniform(1.3, 1.67), pratio=math.exp(r.uniform(1.6, 4.0)))
    elif kind == "sedov":
        control = {} if case["eul"] else dict(kappa=0.01, pmerit=0.1)
        deck = configs.sedov(case["nx"], time_end=1.0e3, eulerian=case["eul"],
                             gamma=r.uniform(1.3, 1.67), energy=r.uniform(0.2, 0.3), **control)
    elif kind in ("noh", "polar"):
        deck = (configs.noh(case["nx"], 1.0e3, case["eul"]) if kind == "noh"
                else configs.noh_polar(case["nx"], case["ny"], 1.0e3))
        deck = deck.replace("density(1)=1.0\n", "density(1)=%r\n" % r.uniform(0.5, 2.0))
        deck = deck.replace("kinematic_param(1,1)=-1.0", "kinematic_param(1,1)=%r" % -r.uniform(0.8, 1.2))
    else:
        s = r.uniform(0.45, 0.6)
        deck, frac = configs.sod_interface(case["nx"], case["ny"], time_end=1.0e3, amplitude=0.0,
                                           periods=0, tilt=case["tilt"], rho_right=s, p_right=s)
    return Problem.from_deck(deck, material_fraction=frac)


def _problems(case, seed):
    if case["kind"] != "ensemble":
        return [_problem(case, seed)]
    # half Sod, half Sedov as configs.ensemble has them: the sizes are the
    # case's, gamma and pressure ratio the seed's
    sides, r = random.Random(case["meshes"] * 1000 + case["nx"] + case["ny"]), random.Random(seed)
    out = []
    for i in range(case["meshes"]):
        side = _logint(sides, case["nx"], case["ny"])
        gamma = r.uniform(1.2, 1.8)
        if i % 2 == 0:
            deck = configs.sod(max(4, round(side * math.sqrt(10.0))), max(2, round(side / math.sqrt(10.0))),
                               time_end=1.0e3, eulerian=case["eul"], gamma=gamma,
                               pratio=math.exp(r.uniform(math.log(2.0), math.log(1.0e4))))
        else:
            deck = configs.sedov(side, time_end=1.0e3, eulerian=case["eul"], gamma=gamma)
        if not case["eul"]:
            deck = deck.replace("cvisc2=0.75\n", "cvisc2=0.75\n kappaall=0.01\n pmeritall=0.1\n")
        out.append(Problem.from_deck(deck))
    return out


class _Host:
    """A host program's arrays of its problems, in one pinned buffer: field
    after field, within a field mesh after mesh (positions and velocities:
    both components of a mesh together), and the initial contents to start
    the next job from."""

    GROUPS = {"position": (abi.NDX, abi.NDY), "velocity": (abi.NDU, abi.NDV)}
    FIELDS = (abi.ELDENSITY, abi.ELENERGY, abi.ELPRESSURE, abi.ELCS2, abi.ELVOLUME, abi.ELVISC)
    CPFIELDS = (abi.CPDENSITY, abi.CPENERGY, abi.FRVOLUME)

    def __init__(self, problems):
        self.problems = problems
        groups = dict(self.GROUPS)
        for f in problems[0].fields:
            if not any(f in g for g in self.GROUPS.values()):
                groups[abi.NAMES[f]] = (f,)
        size = lambda a: -(-a.nbytes // 8)
        total = sum(size(p.fields[f]) for p in problems for g in groups.values() for f in g)
        self.now = torch.empty(total, dtype=torch.float64, pin_memory=True)
        raw, at = self.now.numpy(), 0
        self.whole = {}
        for name, group in groups.items():
            begin = at
            for p in problems:
                for f in group:
                    a = p.fields[f]
                    v = raw[at:at + size(a)].view(a.dtype)[:a.size].reshape(a.shape)
                    v[...] = a
                    p.fields[f] = v
                    at += size(a)
            self.whole[name] = raw[begin:at]
        self.first = self.now.clone()
        self.times = [p.timestep.copy() for p in problems]

    def restore(self):
        self.now.copy_(self.first)
        for p, t in zip(self.problems, self.times):
            for name, _ in t._fields_:
                setattr(p.timestep, name, getattr(t, name))

    def outputs(self, eul):
        """Every mesh's fields, its time, time step and step count."""
        names = list(self.GROUPS) + [abi.NAMES[f] for f in self.FIELDS]
        if eul:
            names += ["elmass", "cnmass"]
        if self.problems[0].sizes.ncp > 0:
            names += [abi.NAMES[f] for f in self.CPFIELDS]
        out = {name: self.whole[name] for name in names}
        ts = [p.timestep for p in self.problems]
        out["time"], out["dt"] = np.array([t.time for t in ts]), np.array([t.dt for t in ts])
        out["nstep"] = np.array([t.nstep for t in ts])
        return out


def _network(seed):
    """A small closure network and the standardisation of its features, of
    the sizes that training gives on such tubes."""
    params = init_params(seed)
    params[-130:] *= 0.2
    mean = np.array([0.5, 0.9, 0.5, 0.8, 0.5, 1.2, 1.5, 0.0, 0.3, 0.2])
    spread = np.array([0.3, 0.3, 0.2, 0.3, 0.2, 0.4, 0.5, 0.01, 0.2, 0.3])
    return params, np.concatenate([mean, 1.0 / spread, [2.0e-4, 3.0]]).astype(np.float32)


def _samples(case, seed):
    """Features and targets like the sub-cell samples': smooth targets that
    nearly cancel."""
    g = np.random.default_rng(seed)
    x = g.normal(0.0, 1.0, (case["samples"], 10)).astype(np.float32)
    t = np.tanh(x[:, :1] * x[:, 1:2] + 0.5 * x[:, 2:3]) + 0.1 * g.normal(size=(len(x), 1))
    return x, np.concatenate([t, -t], axis=1).astype(np.float32)


def prepare(case, seed):
    if case["kind"] == "train":
        x, t = _samples(case, seed)
        return dict(case=case, seed=seed, x=x, t=t, params=init_params(seed))
    host = _Host(_problems(case, seed))
    state = dict(case=case, host=host, solver=None, net=None)
    if case["kind"] == "sod2mat":
        params, state["norm"] = _network(seed)
        state["net"] = ClosureNet(params)
    if case["drive"] != "job":
        state["solver"] = _solver(state)
    return state


def _solver(state):
    case, host = state["case"], state["host"]
    mode = MODES[case["mode"]]
    s = (BatchSolver(host.problems, fp_mode=mode) if case["drive"] == "batch"
         else Solver(host.problems[0], fp_mode=mode))
    if state["net"] is not None:
        s.set_closure(state["net"], state["norm"], volume_only=True)
    return s


# ------------------------------------------------------------------ a pass

def run(state):
    case = state["case"]
    if case["kind"] == "train":
        net = ClosureNet(state["params"])
        losses = net.train(state["x"], state["t"], epochs=case["epochs"], batch=case["batch"],
                           seed=state["seed"])
        out = {"params": net.params(), "losses": losses, "predicted": net.predict(state["x"])}
        net.close()
        return out
    host = state["host"]
    host.restore()
    if case["drive"] == "job":
        s = _solver(state)
    else:
        s = state["solver"]
        s.sync_to_device(0)
    if case["drive"] in ("loop", "batch"):
        rest = s.run(case["steps"]) if case["drive"] == "batch" else s.run(case["steps"], history=False)
        if rest[0] != 0:
            raise RuntimeError(s.error.message)
    else:
        for _ in range(case["steps"]):
            if s.step() != 0:
                raise RuntimeError(s.error.message)
    s.sync_to_host(0)
    if case["drive"] == "job":
        s.close()
    return host.outputs(case["eul"])


def work(case):
    if case["kind"] == "train":
        n = case["samples"]
        return {"bytes": n * 4 * (12 * case["epochs"] + 12),
                "flops": n * 2 * 4864 * (3 * case["epochs"] + 1)}
    if case["kind"] == "ensemble":
        lo, hi = case["nx"], case["ny"]
        cells = case["meshes"] * (hi * hi - lo * lo) / (2.0 * math.log(hi / lo))
    else:
        cells = case["nx"] * case["ny"]
    zc = cells * case["steps"]
    # the fields in and out once, and the steps
    return {"bytes": zc * (EUL_BYTES if case["eul"] else LAG_BYTES) + cells * 800,
            "flops": zc * (EUL_FLOPS if case["eul"] else LAG_FLOPS)}


# ------------------------------------------------------------------ exact

def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    problems = _problems(case, seed)
    sim = _Reference(problems)
    for _ in range(case["steps"]):
        sim.step()
    flat = lambda t: t.reshape(-1).cpu().numpy()
    mine = (sim.rho, sim.e, sim.p, sim.cs2, sim.vol, sim.visc)
    out = {abi.NAMES[f]: flat(t) for f, t in zip(_Host.FIELDS, mine)}
    nodes = [slice(int(a), int(b)) for a, b in zip(sim.nnd[:-1], sim.nnd[1:])]
    for name, (p, q) in (("position", (sim.x, sim.y)), ("velocity", (sim.u, sim.v))):
        out[name] = flat(torch.cat([w[nd] for nd in nodes for w in (p, q)]))
    if case["eul"]:
        out["elmass"], out["cnmass"] = flat(sim.mass), flat(sim.cnmass)
    if problems[0].sizes.ncp > 0:  # what the network decides has no such value
        out.update({abi.NAMES[f]: None for f in _Host.CPFIELDS})
    out["time"], out["dt"] = flat(sim.time), flat(sim.dt)
    out["nstep"] = np.full(len(problems), sim.nstep)
    return out


def _exact_train(case, seed):
    """The training in FP64: the same shuffles, the same Adam."""
    x, t = _samples(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    X, T = torch.tensor(x, dtype=torch.float64, device=dev), torch.tensor(t, dtype=torch.float64, device=dev)
    P = torch.tensor(init_params(seed), dtype=torch.float64, device=dev)
    cut = np.cumsum([640, 64, 4096, 64, 128, 2])

    def net(P, x):
        w1, b1, w2, b2, w3, b3 = (P[a:b] for a, b in zip([0] + list(cut[:-1]), cut))
        z = x @ w1.view(64, 10).T + b1
        z = (z * torch.sigmoid(z)) @ w2.view(64, 64).T + b2
        return (z * torch.sigmoid(z)) @ w3.view(2, 64).T + b3

    n, size = len(x), case["batch"]
    perm = list(range(n))
    mask = (1 << 64) - 1
    r = (seed * 0x9E3779B97F4A7C15 + 1) & mask
    m, v, step, losses = torch.zeros_like(P), torch.zeros_like(P), 0, []
    for _ in range(case["epochs"]):
        for i in range(n - 1, 0, -1):
            r = (r + 0x9E3779B97F4A7C15) & mask
            z = ((r ^ (r >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            z ^= z >> 31
            j = z % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        order = torch.tensor(perm, device=dev)
        total = 0.0
        for at in range(0, n, size):
            at_idx = order[at:at + size]
            Q = P.detach().requires_grad_(True)
            loss = ((net(Q, X[at_idx]) - T[at_idx]) ** 2).sum() / (2 * len(at_idx))
            g, = torch.autograd.grad(loss, Q)
            step += 1
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            P = P - 1e-3 * (m / (1 - 0.9 ** step)) / (torch.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
            total += float(loss) * len(at_idx)
        losses.append(total / n)
    return {"params": P.cpu().numpy(), "losses": np.array(losses), "predicted": net(P, X).cpu().numpy()}


class _Reference:
    """The method over whole-mesh arrays in FP64: edge viscosity, time step,
    predictor and corrector, Eulerian remap, two-material mixed cells under
    the plain closure, ideal gases; several disconnected meshes at once, each
    with its own time step."""

    def __init__(self, problems):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        cat = lambda f: torch.tensor(np.concatenate([p.fields[f] for p in problems]), device=dev)
        nel = np.cumsum([0] + [p.nel for p in problems])
        nnd = np.cumsum([0] + [p.nnd for p in problems])
        self.nel, self.nnd = nel, nnd
        part = lambda f, off: torch.tensor(np.concatenate(
            [p.fields[f].astype(np.int64) - 1 + o for p, o in zip(problems, off)]), device=dev)
        self.nd, self.nb = part(abi.IELND, nnd), part(abi.IELEL, nel)
        self.fc = part(abi.IELFC, [0] * len(problems))
        self.ntype = cat(abi.INDTYPE)
        self.x, self.y, self.u, self.v = (cat(f) for f in (abi.NDX, abi.NDY, abi.NDU, abi.NDV))
        (self.rho, self.e, self.p, self.cs2, self.vol, self.mass, self.visc) = (cat(f) for f in (
            abi.ELDENSITY, abi.ELENERGY, abi.ELPRESSURE, abi.ELCS2, abi.ELVOLUME, abi.ELMASS,
            abi.ELVISC))
        self.a1, self.a2, self.a3, self.b1, self.b2, self.b3 = (cat(f) for f in (
            abi.A1, abi.A2, abi.A3, abi.B1, abi.B2, abi.B3))
        self.cnwt, self.cnmass = cat(abi.CNWT), cat(abi.CNMASS)
        c = self.c = problems[0].config
        self.spmass = cat(abi.SPMASS) if c.zsp else None
        row = lambda get: torch.tensor([get(p) for p in problems], dtype=torch.float64, device=dev)
        self.inst = torch.repeat_interleave(torch.arange(len(problems), device=dev),
                                            torch.tensor(np.diff(nel), device=dev))
        self.ninst = torch.repeat_interleave(torch.arange(len(problems), device=dev),
                                             torch.tensor(np.diff(nnd), device=dev))
        self.time, self.dt = row(lambda p: p.timestep.time), row(lambda p: p.timestep.dt)
        self.dt_g, self.dt_max, self.dt_ini = (row(lambda p: getattr(p.config, k))
                                               for k in ("dt_g", "dt_max", "dt_initial"))
        self.gamma = torch.tensor([[0.0] + [p.config.eos_param[m][0] for m in range(1, 3)]
                                   for p in problems], dtype=torch.float64, device=dev)
        self.mat = cat(abi.IELMAT).long().clamp(min=0)
        self.nstep = 0
        self.ncp = problems[0].sizes.ncp if len(problems) == 1 else 0
        if self.ncp:
            p = problems[0]
            n = p.fields[abi.IMXNCP].astype(np.int64)
            self.cpel = torch.tensor(np.repeat(p.fields[abi.IMXEL].astype(np.int64) - 1, n), device=dev)
            self.cpmat = cat(abi.ICPMAT).long()
            self.cpe, self.cpp, self.cpcs2, self.cpm, self.frv, self.frm = (cat(f) for f in (
                abi.CPENERGY, abi.CPPRESSURE, abi.CPCS2, abi.CPMASS, abi.FRVOLUME, abi.FRMASS))

    def eos(self, g, rho, e):
        p = e * rho * (g - 1.0)
        p = torch.where(p.abs() < self.c.pcut, torch.zeros_like(p), p)
        return p, (g * (g - 1.0) * e).clamp(min=self.c.ccut)

    def el_eos(self, rho, e):
        g = self.gamma[self.inst, self.mat]
        p, c = self.eos(g, rho, e)
        void = self.mat == 0
        p0 = self.c.eos_param[0][0]
        return (torch.where(void, torch.full_like(p, p0 if abs(p0) >= self.c.pcut else 0.0), p),
                torch.where(void, torch.full_like(c, self.c.ccut), c))

    @staticmethod
    def iso(x, y):
        def abc(q):
            q0, q1, q2, q3 = q.unbind(1)
            return 0.25 * (-q0 + q1 + q2 - q3), 0.25 * (q0 - q1 + q2 - q3), 0.25 * (-q0 - q1 + q2 + q3)
        a1, a2, a3 = abc(x)
        b1, b2, b3 = abc(y)
        w = []
        for s1, s3 in ((-1, -1), (-1, 1), (1, 1), (1, -1)):  # (3a1 + s1 a2), (3b3 + s3 b2)
            w.append(((3 * b3 + s3 * b2) * (3 * a1 + s1 * a2) - (3 * a3 + s3 * a2) * (3 * b1 + s1 * b2)) / 9.0)
        return a1, a2, a3, b1, b2, b3, torch.stack(w, 1), 4.0 * (a1 * b3 - a3 * b1)

    @staticmethod
    def sign(a, b):
        return torch.copysign(a, b)

    def viscosity(self):
        """hydro_kn_edgeviscosity: element viscosity and corner forces."""
        zc, nd, nb = self.c.zerocut, self.nd, self.nb
        me = torch.arange(len(nd), device=nd.device)
        x, y, u, v = self.x[nd], self.y[nd], self.u[nd], self.v[nd]
        xc, yc = x.mean(1), y.mean(1)
        visc = torch.zeros_like(self.rho)
        ex, ey = [None] * 4, [None] * 4
        bnd = self.ntype[nd] < 0
        for s in (0, 1):
            n1, n2 = nb[:, s], nb[:, s + 2]
            f1, f2 = self.fc[:, s], self.fc[:, s + 2]
            val1 = (bnd[:, s] & bnd[:, s + 1] & (n2 != me)).double()
            val2 = (bnd[:, s + 2] & bnd[:, (s + 3) % 4] & (n1 != me)).double()
            for k, i in enumerate(((s + 3) % 4, s + 1)):
                j = (i + 1) % 4
                du, dv, dx, dy = u[:, j] - u[:, i], v[:, j] - v[:, i], x[:, j] - x[:, i], y[:, j] - y[:, i]
                lu, lx = torch.sqrt(du * du + dv * dv), torch.sqrt(dx * dx + dy * dy)
                uh, vh = du / lu.clamp(min=zc), dv / lu.clamp(min=zc)
                xh, yh = dx / lx.clamp(min=zc), dy / lx.clamp(min=zc)
                den = dx * xh + dy * yh
                w = (du * uh + dv * vh) / self.sign(den.abs().clamp(min=zc), den)
                w = 1.0 / self.sign(w.abs().clamp(min=zc), w)

                def ratio(n, f, val):
                    a = torch.gather(nd[n], 1, f[:, None])[:, 0]
                    b = torch.gather(nd[n], 1, ((f + 1) % 4)[:, None])[:, 0]
                    d = (self.x[b] - self.x[a]) * xh + (self.y[b] - self.y[a]) * yh
                    q = (self.u[b] - self.u[a]) * uh + (self.v[b] - self.v[a]) * vh
                    q = q / self.sign(d.abs().clamp(min=zc), d) * w
                    return torch.where(n == me, val, q)

                r1 = ratio(n1, (f1 + (1 if k == 0 else 3)) % 4, val1)
                r2 = ratio(n2, (f2 + (3 if k == 0 else 1)) % 4, val2)
                lim = torch.minimum(torch.minimum(0.5 * (r1 + r2), 2 * r1), 2 * r2).clamp(0.0, 1.0)
                other = nb[:, i]
                c = self.c.cvisc1 * torch.sqrt(0.5 * (self.cs2 + self.cs2[other]))
                edv = 0.5 * (1.0 - lim) * (self.rho + self.rho[other]) * (c + self.c.cvisc2 * lu)
                visc = torch.maximum(visc, edv * 2.0 * lu / self.rho.clamp(min=zc))
                mx, my = 0.5 * (x[:, i] + x[:, j]), 0.5 * (y[:, i] + y[:, j])
                w7 = torch.sqrt((xc - mx) ** 2 + (yc - my) ** 2)
                hx, hy = (yc - my) / w7, (mx - xc) / w7
                t = -torch.copysign(w7, hx * xh + hy * yh)
                hx, hy = hx * t, hy * t
                w6 = du * hx + dv * hy
                d = edv * (w6 / lu.clamp(min=zc))
                cut = (lu <= zc) | (w6 <= zc) | (w7 <= zc) | (lx <= zc)
                ex[i] = torch.where(cut, torch.zeros_like(d), du * d)
                ey[i] = torch.where(cut, torch.zeros_like(d), dv * d)
        corner = lambda e: torch.stack([e[0] - e[3], e[1] - e[0], e[2] - e[1], e[3] - e[2]], 1)
        return visc, corner(ex), corner(ey)

    def getdt(self):
        self.visc, self.qx, self.qy = self.viscosity()
        x, y, u, v = self.x[self.nd], self.y[self.nd], self.u[self.nd], self.v[self.nd]
        self.cs2v = self.cs2 + self.visc
        if self.ncp:
            s = torch.zeros_like(self.cs2v).index_add(0, self.cpel, self.frm * self.cpcs2)
            mixed = torch.zeros_like(self.cs2v, dtype=torch.bool)
            mixed[self.cpel] = True
            self.cs2v = torch.where(mixed, s, self.cs2v)
        best = None
        for k in range(4):
            a, b, c, d = k, (k + 1) % 4, (k + 2) % 4, (k + 3) % 4
            w1 = (x[:, c] - x[:, d]) ** 2 + (y[:, c] - y[:, d]) ** 2
            pp = (0.5 * (x[:, a] + x[:, b]) - x[:, c]) ** 2 + (0.5 * (y[:, a] + y[:, b]) - y[:, c]) ** 2
            # twice the triangle (edge c-d, midpoint of a-b)
            area = ((x[:, d] - x[:, c]) * (0.5 * (y[:, a] + y[:, b]) - y[:, c])
                    - (y[:, d] - y[:, c]) * (0.5 * (x[:, a] + x[:, b]) - x[:, c]))
            r = torch.where(w1 < self.c.zcut, pp, area * area / w1)
            best = r if best is None else torch.minimum(best, r)
        n = len(self.dt)
        new = lambda fill: torch.full((n,), fill, dtype=torch.float64, device=x.device)
        cfl = new(math.inf).scatter_reduce(0, self.inst, best / self.cs2v, "amin")
        w = (u[:, 0] - u[:, 2]) * (self.b1 - self.b3) + (u[:, 1] - u[:, 3]) * (self.b1 + self.b3) \
            - (v[:, 0] - v[:, 2]) * (self.a1 - self.a3) - (v[:, 1] - v[:, 3]) * (self.a1 + self.a3)
        div = new(2.2250738585072014e-308).scatter_reduce(0, self.inst, w.abs() / self.vol, "amax")
        dt = torch.minimum(self.dt_max, self.dt_g * self.dt)
        if self.nstep == 0:
            dt = torch.minimum(dt, self.dt_ini)
        dt = torch.minimum(torch.minimum(dt, self.c.cfl_sf * torch.sqrt(cfl)), self.c.div_sf / div)
        self.dt, self.time, self.nstep = dt, self.time + dt, self.nstep + 1

    @staticmethod
    def pressure(p, a1, a3, b1, b3):
        fx = torch.stack([b1 - b3, b3 + b1, b3 - b1, -b3 - b1], 1) * p[:, None]
        fy = torch.stack([a3 - a1, -a3 - a1, a1 - a3, a3 + a1], 1) * p[:, None]
        return fx, fy

    def subzonal(self, w1, rho, cs2, x, y):
        xm, ym = x.mean(1), y.mean(1)
        lx, ly = [], []
        mid = lambda q, j: 0.5 * (q[:, j] + q[:, (j + 1) % 4])
        for j in range(4):
            X = torch.stack([x[:, j], mid(x, j), xm, mid(x, (j + 3) % 4)], 1)
            Y = torch.stack([y[:, j], mid(y, j), ym, mid(y, (j + 3) % 4)], 1)
            a1, _, a3, b1, _, b3, _, vol = self.iso(X, Y)
            fx, fy = self.pressure(cs2 * (self.spmass[:, j] / vol - rho), a1, a3, b1, b3)
            lx.append(fx)
            ly.append(fy)
        out = []
        for l in (lx, ly):
            c = 0.25 * (l[0][:, 2] + l[1][:, 2] + l[2][:, 2] + l[3][:, 2])
            m = [0.5 * (l[j][:, 1] + l[(j + 1) % 4][:, 3]) for j in range(4)]
            out.append(torch.stack([w1 * (l[j][:, 0] + m[j] + m[(j + 3) % 4] + c) for j in range(4)], 1))
        return out

    def lagstep(self):
        c, nd, zc = self.c, self.nd, self.c.zerocut
        x, y, u, v = self.x[nd], self.y[nd], self.u[nd], self.v[nd]
        dt = self.dt[self.inst]
        mass = self.mass.clamp(min=zc)
        region = 0  # the controls are the same in every region here
        fx, fy = self.pressure(self.p, self.a1, self.a3, self.b1, self.b3)
        fx, fy = fx + self.qx, fy + self.qy
        if c.zsp:
            sx, sy = self.subzonal(c.pmeritreg[region], self.rho, self.cs2v, x, y)
            fx, fy = fx + sx, fy + sy
        half = 0.5 * dt
        a1, _, a3, b1, _, b3, w, vol = self.iso(x + half[:, None] * u, y + half[:, None] * v)
        rho = self.mass / vol
        e = self.e - (fx * u + fy * v).sum(1) / mass * half
        p, cs2 = self.el_eos(rho, e)
        gx, gy = self.pressure(p, a1, a3, b1, b3)
        gx, gy = gx + self.qx, gy + self.qy
        if c.zsp:
            sx, sy = self.subzonal(c.pmeritreg[region], rho, cs2, x + half[:, None] * u,
                                   y + half[:, None] * v)
            gx, gy = gx + sx, gy + sy
        if c.zhg:
            alt = torch.tensor([1.0, -1.0, 1.0, -1.0], dtype=torch.float64, device=x.device)
            k = (-c.kappareg[region] * rho * vol / dt)[:, None] * alt
            gx, gy = gx + k * (u * alt).sum(1, keepdim=True), gy + k * (v * alt).sum(1, keepdim=True)
        if self.ncp:
            ce, cm = self.cpel, self.cpm.clamp(min=zc)
            fr = self.frv[:, None]
            hx, hy = self.pressure(self.cpp, self.a1[ce], self.a3[ce], self.b1[ce], self.b3[ce])
            self.cpe = self.cpe - (hx * fr * u[ce] + hy * fr * v[ce]).sum(1) / cm * half[ce]
            g = self.gamma[0, self.cpmat]
            cp, _ = self.eos(g, self.cpm / (vol[ce] * self.frv), self.cpe)
            hx, hy = self.pressure(cp, a1[ce], a3[ce], b1[ce], b3[ce])
            gx[ce], gy[ce] = 0.0, 0.0
            gx, gy = gx.index_add(0, ce, fr * hx), gy.index_add(0, ce, fr * hy)
        # nodes
        zero = torch.zeros_like(self.x)
        scatter = lambda q: zero.index_add(0, nd.reshape(-1), q.reshape(-1))
        prev = self.cnmass[:, [3, 0, 1, 2]]
        m = torch.where(self.cnmass > zc, self.cnmass, torch.where(prev > zc, prev, rho[:, None] * w))
        m, area = scatter(m), scatter(w)
        ok = m > c.dencut * area
        safe = torch.where(ok, m, torch.ones_like(m))
        ax, ay = (torch.where(ok, scatter(q) / safe, zero) for q in (gx, gy))
        t = self.ntype
        ax = torch.where((t == -1) | (t == -3), zero, ax)
        ay = torch.where((t == -2) | (t == -3), zero, ay)
        low = ax * ax + ay * ay < c.accut * c.accut
        ax, ay = torch.where(low, zero, ax), torch.where(low, zero, ay)
        ndt = self.dt[self.ninst]
        u1, v1 = self.u + ndt * ax, self.v + ndt * ay
        self.ub, self.vb = 0.5 * (self.u + u1), 0.5 * (self.v + v1)
        self.x, self.y = self.x + ndt * self.ub, self.y + ndt * self.vb
        self.u, self.v = u1, v1
        ub, vb = self.ub[nd], self.vb[nd]
        self.geometry()
        self.rho = self.mass / self.vol
        self.e = self.e - (gx * ub + gy * vb).sum(1) / mass * dt
        self.p, self.cs2 = self.el_eos(self.rho, self.e)
        if self.ncp:
            self.cpe = self.cpe - (hx * fr * ub[ce] + hy * fr * vb[ce]).sum(1) / cm * dt[ce]
            self.cpp, self.cpcs2 = self.eos(g, self.cpm / (self.vol[ce] * self.frv), self.cpe)

    def geometry(self):
        (self.a1, self.a2, self.a3, self.b1, self.b2, self.b3, self.cnwt, self.vol) = self.iso(
            self.x[self.nd], self.y[self.nd])

    def limited(self, basis, flux, var):
        """Limited flux of an element variable through each face."""
        nb, fc, out = self.nb, self.fc, [None] * 4
        at = lambda n, f: (torch.gather(basis[n], 1, f[:, None])
                           + torch.gather(basis[n], 1, ((f + 1) % 4)[:, None]))[:, 0]
        for i in (0, 1):
            j = i + 2
            r3 = basis[:, j] + basis[:, (j + 1) % 4]
            r4 = basis[:, i] + basis[:, i + 1]
            w5, w6 = r3 + at(nb[:, j], fc[:, j]), r4 + at(nb[:, i], fc[:, i])
            w1, w2 = var - var[nb[:, j]], var[nb[:, i]] - var
            g = self.slope(w1, w2, w5, w6)
            out[i] = flux[:, i] * (var + g * (r3 - 0.5 * flux[:, i]))
            out[j] = flux[:, j] * (var - g * (r4 - 0.5 * flux[:, j]))
        return torch.stack(out, 1)

    def slope(self, w1, w2, w5, w6):
        w8 = (w1 * w6 * w6 + w2 * w5 * w5) / (w5 * w6 * (w5 + w6))
        g = torch.minimum(torch.minimum(w8.abs(), w1.abs() / w5), w2.abs() / w6)
        return torch.where(w1 * w2 <= 0.0, torch.zeros_like(g), torch.copysign(g, w2))

    def inflow(self, flux):
        """Each face's flux as the neighbour has it (0 at a boundary)."""
        me = torch.arange(len(self.nb), device=self.nb.device)
        q = torch.stack([torch.gather(flux[self.nb[:, f]], 1, self.fc[:, f:f + 1])[:, 0] for f in range(4)], 1)
        return torch.where(self.nb == me[:, None], torch.zeros_like(q), q)

    def alestep(self):
        nd, nb, fc, zc = self.nd, self.nb, self.fc, self.c.zerocut
        ndt = self.dt[self.ninst]
        x0, y0 = self.x[nd], self.y[nd]
        xn, yn = self.x - ndt * self.ub, self.y - ndt * self.vb
        x1, y1 = xn[nd], yn[nd]
        fv = []
        for j in range(4):
            k = (j + 1) % 4
            # the quadrilateral the face sweeps, by its diagonals' cross product
            d1x, d1y = x1[:, k] - x0[:, j], y1[:, k] - y0[:, j]
            d2x, d2y = x1[:, j] - x0[:, k], y1[:, j] - y0[:, k]
            d = 0.5 * (d1x * d2y - d1y * d2x)
            fv.append(torch.where(d < zc, torch.zeros_like(d), d))
        fv = torch.stack(fv, 1)
        fm = self.limited(self.cnwt, fv, self.rho)
        nfm = self.inflow(fm)
        vpr, mpr = self.vol, self.mass
        self.mass = mpr + (nfm - fm).sum(1)
        ef = self.limited(self.cnmass, fm, self.e)
        net = nfm - fm
        cb = [0.25 * (net[:, i % 2] - net[:, i % 2 + 2]) for i in range(4)]
        cflux = 0.25 * net.sum(1)
        u, v = self.u[nd], self.v[nd]
        ob, fu, fw = self.cnmass, [0.0] * 4, [0.0] * 4
        for l in (0, 1):
            r = l + 2
            fl, fr = fc[:, l] + 1, fc[:, r] + 1
            for n in (1, 2):
                a, b = l + n - 1, (r + 2 - n) % 4
                cd = cb[l + 2 * (n - 1)]
                left = cd > 0
                el = torch.where(left, nb[:, l], nb[:, r])
                nl = torch.where(left, (fl + n) % 4, (fr + n - 2) % 4)
                nr = torch.where(left, (fl - n + 1) % 4, (fr - n - 1) % 4)
                far = torch.gather(nd[el], 1, torch.where(left, nl, nr)[:, None])[:, 0]
                w5 = ob[:, a] + ob[:, b]
                w6 = (torch.gather(ob[el], 1, nl[:, None]) + torch.gather(ob[el], 1, nr[:, None]))[:, 0]
                dist = torch.where(left, ob[:, a], ob[:, b]) - 0.5 * cd.abs()
                for var, cv, f in ((self.u, u, fu), (self.v, v, fw)):
                    near = torch.where(left, cv[:, a], cv[:, b])
                    inner = torch.where(left, cv[:, b], cv[:, a]) - near
                    outer = near - var[far]
                    d = cd * (near + self.slope(inner, outer, w5, w6) * dist)
                    d = torch.where(cd == 0, torch.zeros_like(d), d)
                    f[a], f[b] = f[a] - d, f[b] + d
        fu, fw = torch.stack(fu, 1), torch.stack(fw, 1)
        zero = torch.zeros_like(self.x)
        scatter = lambda q: zero.index_add(0, nd.reshape(-1), q.reshape(-1))
        m0 = scatter(self.cnmass)
        m1 = m0 + scatter(cflux[:, None].expand(-1, 4))
        ok = m1 > self.c.dencut * scatter(0.25 * vpr[:, None].expand(-1, 4))
        safe = torch.where(ok, m1, torch.ones_like(m1))
        t = self.ntype
        self.u = torch.where(ok & (t != -1) & (t != -3), (self.u * m0 + scatter(fu)) / safe, self.u)
        self.v = torch.where(ok & (t != -2) & (t != -3), (self.v * m0 + scatter(fw)) / safe, self.v)
        self.x, self.y = xn, yn
        moved = self.mass > vpr * self.c.dencut
        gain = (self.inflow(ef) - ef).sum(1)
        self.e = torch.where(moved, (self.e * mpr + gain) / torch.where(moved, self.mass, torch.ones_like(mpr)), self.e)
        self.cnmass = self.cnmass + cflux[:, None]
        self.geometry()
        self.rho = self.mass / self.vol
        self.p, self.cs2 = self.el_eos(self.rho, self.e)

    def step(self):
        self.getdt()
        self.lagstep()
        if self.c.ale_zexist:
            self.alestep()
