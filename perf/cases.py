"""The calls that a program using this framework makes, as cases that can be timed and checked.

Every case goes through the public Python classes (``BatchedFiberRVEAnalysisExplicit``,
``MicroFOBatch``, ``RVEServer``). Networks come from the package's seeded generator, with the sizes,
material distributions and deformation gradients of the configurations in
``mumfim_gb300/synthetic.py``; step counts are shorter than there (every step costs the same), so
that a pass takes milliseconds. ``exact`` solves the same inputs with plain torch in 64 bits.

A case's values:

  call       what one pass calls:
               run        run(F, sigma, update_coords=False): host arrays in and out
               device     run_device() on device-resident F and sigma, not updating
               cycle      a load increment and its inverse as two updating runs, then the
                          displacements of every RVE
               stiffness  computeMaterialStiffness() after an updating run
               couple     a load increment and its inverse as two micro_fo iterations (stress and
                          stiffness), then the step results (orientation tensors)
               serve      every RVE's load increment and its inverse submitted to a server, drained
  precision  "f64" or "mixed"
  law        "linear", "nonlinear" or "both" (alternating)
  mode       "ramp" (fixed number of steps) or "relax" (until the residual is small, at most `steps`)
  rves, n_min, n_max, k, steps
             number of RVEs, their node counts (log-uniform), fibers per node of the generator
             (0: 3, 4 and 5 in turn), explicit steps of one solve
"""
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import mumfim_gb300 as m
from mumfim_gb300 import synthetic
from mumfim_gb300.coupling import MicroFOBatch
from mumfim_gb300.network_io import LINEAR, NONLINEAR, Reaction
from mumfim_gb300.serving import RVEServer


def _case(name, call, precision, law, mode, rves, n_min, n_max, k, steps):
    return {"name": name, "call": call, "precision": precision, "law": law, "mode": mode,
            "rves": rves, "n_min": n_min, "n_max": n_max, "k": k, "steps": steps}


def listed():
    return [
        # one RVE of 1000 nodes, as someone checking a network alone runs it: latency of a step
        _case("single_f64", "run", "f64", "linear", "ramp", 1, 1000, 1000, 4, 1000),
        # a handful of small relaxing RVEs with stress, stiffness and orientation: the standalone
        # driver's job and the smallest macro problem
        _case("couple_relax_f64", "couple", "f64", "linear", "relax", 4, 300, 900, 4, 400),
        # many RVEs of one size in plain FP64: the reference's production batch
        _case("uniform_f64", "device", "f64", "linear", "ramp", 256, 4500, 4500, 4, 100),
        # an uneven FP64 batch, both fiber laws: what a mixed-precision run is checked against
        _case("uneven_f64", "run", "f64", "both", "ramp", 64, 500, 20000, 0, 60),
        # one RVE of ordinary size in mixed precision: latency of a step
        _case("single_mixed", "run", "mixed", "linear", "ramp", 1, 4500, 4500, 4, 2000),
        # the integration points of a few macro elements, load steps that update the state
        _case("few_cycle_mixed", "cycle", "mixed", "linear", "ramp", 12, 500, 20000, 0, 500),
        # the uneven production batch
        _case("uneven_mixed", "device", "mixed", "linear", "ramp", 512, 500, 20000, 0, 1000),
        # the exponential-toe law at its sizes
        _case("nonlinear_mixed", "run", "mixed", "nonlinear", "ramp", 192, 2000, 8000, 4, 1000),
        # RVEs larger than a small cluster's shared memory
        _case("large_mixed", "run", "mixed", "linear", "ramp", 3, 25000, 80000, 4, 100),
        # macro iterations over relaxing RVEs: stress, six perturbed solves, orientation tensors
        _case("couple_relax_mixed", "couple", "mixed", "both", "relax", 24, 300, 3000, 4, 200),
        # the tangent of a RAMP batch: six perturbed solves in flight at once
        _case("stiffness_mixed", "stiffness", "mixed", "linear", "ramp", 32, 500, 20000, 0, 200),
        # a wave of increments from a macro solver through the continuous-batching server
        _case("served_mixed", "serve", "mixed", "both", "ramp", 96, 500, 20000, 0, 200),
    ]


# fiber-steps of one pass that a drawn case may have, by precision: no more than the largest listed
_MOST = {"f64": 2.4e8, "mixed": 5.0e9}


def draw(rng):
    call, precision, law, mode, rves, n_lo, n_hi, steps = rng.choice([
        ("run", "f64", "linear", "ramp", (1, 4), 300, 5000, (100, 1000)),
        ("couple", "f64", "linear", "relax", (1, 8), 200, 1500, (100, 400)),
        ("device", "f64", "linear", "ramp", (20, 256), 1000, 6000, (20, 200)),
        ("run", "f64", "both", "ramp", (5, 64), 500, 20000, (20, 60)),
        ("run", "mixed", "linear", "ramp", (1, 6), 500, 20000, (300, 2000)),
        ("cycle", "mixed", "both", "ramp", (2, 40), 500, 20000, (100, 500)),
        ("device", "mixed", "linear", "ramp", (40, 512), 500, 20000, (200, 1000)),
        ("run", "mixed", "nonlinear", "ramp", (4, 192), 500, 8000, (200, 1000)),
        ("run", "mixed", "linear", "ramp", (1, 5), 20000, 80000, (40, 100)),
        ("couple", "mixed", "both", "relax", (2, 48), 200, 4000, (100, 300)),
        ("stiffness", "mixed", "linear", "ramp", (2, 64), 500, 20000, (100, 300)),
        ("serve", "mixed", "both", "ramp", (8, 128), 500, 20000, (100, 400)),
    ])

    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    n_min, n_max = sorted((spread(n_lo, n_hi), spread(n_lo, n_hi)))
    case = {"call": call, "precision": precision, "law": law, "mode": mode,
            "rves": spread(*rves), "n_min": n_min, "n_max": n_max, "k": rng.choice((0, 3, 4, 5)),
            "steps": spread(*steps)}
    while _fibers(case) * _solves(case) * case["steps"] > _MOST[precision]:
        if case["rves"] > 1:
            case["rves"] = max(1, case["rves"] * 2 // 3)
        else:
            case["steps"] = case["steps"] * 2 // 3
    # the largest RVE alone bounds the pass as well
    while n_max * _solves(case) * case["steps"] > (4.0e6 if precision == "f64" else 2.0e7):
        case["steps"] = case["steps"] * 2 // 3
    return case


# ---- inputs -----------------------------------------------------------------------------------

def _sizes(case):
    """Node counts: log-uniform between n_min and n_max, in no order; the same for every seed."""
    at = [(i * 0.6180339887498949 + 0.5) % 1.0 for i in range(case["rves"])]
    return [int(round(case["n_min"] * (case["n_max"] / case["n_min"]) ** t)) for t in at]


def _ks(case):
    return [case["k"] or 3 + i % 3 for i in range(case["rves"])]


def _solves(case):
    return {"run": 1, "device": 1, "cycle": 2, "stiffness": 6, "couple": 14, "serve": 2}[case["call"]]


def _fibers(case):
    """Expected fiber count (the generator keeps about 0.62 k fibers per node)."""
    return sum(0.62 * k * n for n, k in zip(_sizes(case), _ks(case)))


def _inputs(case, seed):
    """(networks, strategies, F): materials and deformation gradients distributed as in the
    package's configurations."""
    rng = np.random.default_rng(seed)
    sizes, ks, nr = _sizes(case), _ks(case), case["rves"]
    relax = case["mode"] == "relax"
    z = rng.standard_normal((nr, 2))
    w = rng.uniform(size=(nr, 13))
    reactions, F = [], np.zeros((nr, 3, 3))
    for i in range(nr):
        nonlinear = case["law"] == "nonlinear" or (case["law"] == "both" and i % 2 == 1)
        B, lt = (1.0 + 9.0 * w[i, 0], 1.02 + 0.13 * w[i, 1]) if nonlinear else (0.0, 0.0)
        if relax:  # the standalone driver's material
            r, E, rho = 5e-5, 1e8 * math.exp(0.3 * z[i, 1]), 1000.0
        else:
            r, E, rho = 1e-3 * math.exp(0.2 * z[i, 0]), math.exp(0.3 * z[i, 1]), 1.0
        reactions.append(Reaction(NONLINEAR if nonlinear else LINEAR, r, E, rho, B, lt))
        if case["law"] == "nonlinear":
            F[i] = np.diag([1.0 + 0.25 * w[i, 2], 1.0, 1.0])
            F[i] = F[i] @ np.array([[1.0, 0.3 * w[i, 3] - 0.15, 0.0], [0, 1, 0], [0, 0, 1]])
        else:
            most = {"couple": 0.01, "serve": 0.005}.get(case["call"], 0.08)
            F[i] = np.eye(3) + most * (2.0 * w[i, 4:].reshape(3, 3) - 1.0)

    def one(i):
        return synthetic.knn_network(sizes[i], ks[i], synthetic.geometry_seed(seed & 0x7FFFFFFF, i))

    with ThreadPoolExecutor(max_workers=16) as ex:
        made = list(ex.map(one, range(nr)))
    networks = [m.FiberNetwork(c, e, [rc]) for (c, e), rc in zip(made, reactions)]
    if relax:
        strategy = m.SolutionStrategy(visc_damp_coeff=100.0, residual_tol=1e-6,
                                      max_steps=case["steps"])
    else:
        strategy = m.SolutionStrategy.ramp(case["steps"], 0.5)
    return networks, [strategy] * nr, F


def _micro_fo_params(networks):
    """micro_fo_params records: radius, volume fraction, modulus, B, transition, axis."""
    return np.array([[n.reactions[0].radius, 0.003, n.reactions[0].youngs_modulus,
                      n.reactions[0].B, n.reactions[0].length_ratio_trns, 1.0, 0.5, 0.25]
                     for n in networks])


def prepare(case, seed):
    networks, strategies, F = _inputs(case, seed)
    call, precision, nr = case["call"], case["precision"], case["rves"]
    state = {"call": call, "rves": nr, "F": F, "back": np.linalg.inv(F)}
    if call == "serve":
        # a short idle timeout: a program that shares the GPU with other work frees it soon
        state["server"] = RVEServer(networks, strategies, precision=precision,
                                    idle_timeout_us=300)
    elif call == "couple":
        state["batch"] = MicroFOBatch(networks, _micro_fo_params(networks), strategies,
                                      precision=precision)
    else:
        state["analysis"] = m.BatchedFiberRVEAnalysisExplicit(networks, strategies,
                                                              precision=precision)
        state["sigma"] = np.zeros((nr, 6))
    if call == "device":
        state["F_dev"] = torch.tensor(F.reshape(nr, 9), device="cuda")
        state["sigma_dev"] = torch.zeros((nr, 6), dtype=torch.float64, device="cuda")
    if call == "stiffness":
        state["analysis"].run(F, state["sigma"])
    return state


def run(state):
    call = state["call"]
    if call == "serve":
        server = state["server"]
        for F in (state["F"], state["back"]):
            for r in range(state["rves"]):
                server.submit(r, F[r])
        done = server.drain()
        done = done[np.argsort(done["ticket"])]
        return {"sigma": done["sigma"], "steps": done["steps"], "status": done["status"]}
    if call == "couple":
        batch = state["batch"]
        there = batch.iterate(state["F"])
        back = batch.iterate(state["back"])
        return {"there": there, "back": back, "step": batch.step_results(),
                "steps": batch.last_status["steps"]}
    analysis, sigma = state["analysis"], state["sigma"]
    if call == "stiffness":
        return {"C": analysis.computeMaterialStiffness()}
    if call == "device":
        analysis.run_device(state["F_dev"].data_ptr(), state["rves"],
                            state["sigma_dev"].data_ptr(), update_coords=False,
                            stream=torch.cuda.current_stream().cuda_stream)
        return {"sigma": state["sigma_dev"]}
    if call == "cycle":
        analysis.run(state["F"], sigma)
        there = sigma.copy()
        analysis.run(state["back"], sigma)
        u = [analysis.displacements(r) for r in range(state["rves"])]
        return {"there": there, "back": sigma.copy(), "u": np.concatenate(u)}
    analysis.run(state["F"], sigma, update_coords=False)
    st = analysis.last_status
    return {"sigma": sigma.copy(), "steps": st["steps"], "status": st["status"],
            "residual": st["residual"]}


def work(case):
    """Bytes: the networks (coordinates 24 B and mass 8 B per node, ends and length 16 B per fiber)
    and the FP64 state (x, u: 48 B per node) read once, the state written once per solve. Flops of
    a step: about 30 per fiber and 35 per node, as the algorithm counts them."""
    nodes, fibers, solves = sum(_sizes(case)), _fibers(case), _solves(case)
    flops = solves * case["steps"] * (30.0 * fibers + 35.0 * nodes)
    return {"bytes": nodes * (32.0 + 48.0 + 48.0 * solves) + 16.0 * fibers, "flops": flops}


# ---- the same in 64 bits ------------------------------------------------------------------------

class _Reference:
    """All RVEs of a case as one graph, advanced together in FP64."""

    def __init__(self, networks, strategies, scale):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.dev, self.R = dev, len(networks)

        def t(x, dtype=torch.float64):
            return torch.as_tensor(np.asarray(x), dtype=dtype, device=dev)

        n = [net.n_nodes for net in networks]
        off = np.concatenate([[0], np.cumsum(n)])
        self.X = t(np.concatenate([net.coords for net in networks]))
        conn = np.concatenate([np.asarray(net.connectivity) + o for net, o in zip(networks, off)])
        self.c0, self.c1 = (t(conn[:, q].astype(np.int64), torch.int64) for q in (0, 1))
        self.node_rve = t(np.repeat(np.arange(self.R), n), torch.int64)
        self.fib_rve = t(np.repeat(np.arange(self.R), [net.n_fibers for net in networks]),
                         torch.int64)
        self.bnd = ((self.X.abs() - 0.5).abs() < 1e-8).any(dim=1)
        rc = [net.reactions[0] for net in networks]
        area = t([r.radius * r.radius * math.pi for r in rc])
        rho, E = t([r.density for r in rc]), t([r.youngs_modulus for r in rc])
        self.sound = (E / rho).sqrt()
        self.EA = (E * area)[self.fib_rve]
        self.nonlinear = t([r.law == 1 for r in rc], torch.bool)[self.fib_rve]
        self.any_nonlinear = bool(self.nonlinear.any())
        self.B = t([r.B if r.law == 1 else 1.0 for r in rc])[self.fib_rve]
        self.lt = t([r.length_ratio_trns if r.law == 1 else 1.0 for r in rc])[self.fib_rve]
        self.l0 = (self.X[self.c1] - self.X[self.c0]).norm(dim=1)
        half = (rho * area)[self.fib_rve] * self.l0 * 0.5
        self.mass = torch.zeros(len(self.X), dtype=torch.float64, device=dev)
        self.mass.index_add_(0, self.c0, half).index_add_(0, self.c1, half)
        self.mass.clamp_(min=1e-300)
        s = strategies[0]
        self.ramp, self.cap, self.tol = s.mode == 1, s.max_steps, s.residual_tol
        self.damp, self.crit = s.visc_damp_coeff, s.crit_time_scale_factor
        self.scale = t(scale)
        self.x, self.u = self.X.clone(), torch.zeros_like(self.X)
        self.vol = torch.ones(self.R, dtype=torch.float64, device=dev)
        self.cur = torch.zeros((self.R, 6), dtype=torch.float64, device=dev)

    def per_rve(self, values, rve):
        return torch.zeros(self.R, dtype=torch.float64, device=self.dev).index_add_(0, rve, values)

    def forces(self):
        """(internal force per node, fiber lengths)."""
        d = self.x[self.c1] - self.x[self.c0]
        length = d.norm(dim=1)
        lam = length / self.l0
        green = 0.5 * (lam * lam - 1.0)
        T = lam * self.EA * green
        if self.any_nonlinear:
            a, B, lt = self.EA / self.B, self.B, self.lt
            e = torch.exp(B * 0.5 * (lt * lt - 1.0))
            beyond = a * ((1.0 + lt * lt * B) * e - 1.0) * (lam - lt) + a * lt * (e - 1.0)
            toe = a * lam * torch.expm1(torch.minimum(B * green, B * 0.5 * (lt * lt - 1.0)))
            law = torch.where(lam > lt, beyond, torch.where(lam < 1.0, a * B * (lam - 1.0), toe))
            T = torch.where(self.nonlinear, law, T)
        t = d * (T / length)[:, None]
        f = torch.zeros_like(self.x).index_add_(0, self.c0, t, alpha=-1.0)
        return f.index_add_(0, self.c1, t), length

    def dt(self, length):
        shortest = torch.full((self.R,), math.inf, dtype=torch.float64, device=self.dev)
        return shortest.scatter_reduce_(0, self.fib_rve, length, "amin") / self.sound

    def solve(self, F, update):
        """One solve; (sigma, residual) per RVE."""
        F = torch.as_tensor(np.broadcast_to(F, (self.R, 3, 3)).copy(), device=self.dev)
        grad = (F - torch.eye(3, dtype=torch.float64, device=self.dev))[self.node_rve]

        def moved(x):
            return (grad @ x[:, :, None])[:, :, 0]

        if update:
            self.vol = self.vol * torch.linalg.det(F)
        up = self.u if self.ramp else self.u + moved(self.x)
        self.x = self.X + up
        start, move = self.x, moved(self.x)
        free = (~self.bnd)[:, None]
        v = torch.zeros_like(self.x)
        f, length = self.forces()
        dt = self.dt(length)
        h_prev = torch.zeros(self.R, dtype=torch.float64, device=self.dev)
        active = torch.ones(self.R, dtype=torch.bool, device=self.dev)
        residual = torch.full((self.R,), 10.0, dtype=torch.float64, device=self.dev)
        for step in range(self.cap + 1):
            if step > 0 and (step - 1) % 100 == 0:
                sq = self.per_rve((f * f).sum(dim=1) * free[:, 0], self.node_rve)
                residual = torch.where(active, sq.sqrt(), residual)
                if not self.ramp:
                    active = active & (residual > self.tol)
                    if not bool(active.any()):
                        break
            if step >= self.cap:
                break
            h = self.crit * dt * 0.5
            total = -f - (self.damp * self.mass)[:, None] * v
            v = v + ((h_prev + h)[self.node_rve] / self.mass)[:, None] * total
            drift = (2.0 * h * active)[self.node_rve][:, None] * v
            x = torch.where(free, self.x + drift, self.x)
            if self.ramp:
                x = torch.where(free, x, start + ((step + 1) / self.cap) * move)
            self.x = x
            f, length = self.forces()
            if step % 100 == 0:
                dt = torch.where(active, self.dt(length), dt)
            h_prev = h
        on = self.bnd[:, None]
        sym = self.x[:, :, None] * (f * on)[:, None, :]
        sym = 0.5 * (sym + sym.transpose(1, 2))
        voigt = torch.stack([sym[:, 0, 0], sym[:, 1, 1], sym[:, 2, 2], sym[:, 1, 2], sym[:, 0, 2],
                             sym[:, 0, 1]], dim=1)
        sigma = torch.zeros((self.R, 6), dtype=torch.float64, device=self.dev)
        sigma = sigma.index_add_(0, self.node_rve, voigt) * (self.scale / self.vol)[:, None]
        if update:
            self.u, self.cur = self.x - self.X, sigma
        return sigma, residual

    def stiffness(self):
        """Finite differences of six perturbed solves, as the path defines them: in RAMP mode
        each starts from the updated state, in RELAX mode from the previous one's coordinates."""
        h = 1e-5
        one = math.sqrt(1.0 / (1.0 - 2.0 * h))
        a, b = math.sqrt((1.0 + h) / (1.0 - h * h)), math.sqrt((1.0 - h) / (1.0 - h * h))
        mean, off = 0.5 * (a + b), 0.5 * (a - b)
        C = torch.zeros((self.R, 6, 6), dtype=torch.float64, device=self.dev)
        for i in range(6):
            F = np.eye(3)
            if i < 3:
                F[i, i] = one
            else:
                p, q = ((1, 2), (0, 2), (0, 1))[i - 3]
                F[p, p] = F[q, q] = mean
                F[p, q] = F[q, p] = off
            C[:, :, i] = (self.solve(F, False)[0] - self.cur) / h
        return C

    def orientation(self, normal=None):
        d = self.x[self.c1] - self.x[self.c0]
        d = d / d.norm(dim=1, keepdim=True)
        if normal is not None:
            nv = torch.as_tensor(normal, device=self.dev)
            nv = (nv / (nv * nv).sum(dim=1, keepdim=True))[self.fib_rve]
            d = d - nv * (d * nv).sum(dim=1, keepdim=True)
            d = d / d.norm(dim=1, keepdim=True)
        outer = (d[:, :, None] * d[:, None, :]).reshape(-1, 9)
        count = self.per_rve(torch.ones_like(self.l0), self.fib_rve)
        total = torch.zeros((self.R, 9), dtype=torch.float64, device=self.dev)
        return total.index_add_(0, self.fib_rve, outer) / count[:, None]


def _scale(networks, params):
    """1 / d^2 with d = sqrt(L pi r^2 / volume fraction), L the total fiber length."""
    out = []
    for net, p in zip(networks, params):
        ends = np.asarray(net.coords)[np.asarray(net.connectivity)]
        total = np.linalg.norm(ends[:, 1] - ends[:, 0], axis=1).sum()
        out.append(p[1] / (total * math.pi * p[0] * p[0]))
    return out


def exact(case, seed):
    networks, strategies, F = _inputs(case, seed)
    back, call = np.linalg.inv(F), case["call"]
    params = _micro_fo_params(networks)
    ref = _Reference(networks, strategies,
                     _scale(networks, params) if call == "couple" else [1.0] * case["rves"])
    if call == "serve":
        sigma = torch.cat([ref.solve(F, True)[0], ref.solve(back, True)[0]])
        return {"sigma": sigma, "steps": None, "status": None}
    if call == "couple":
        got = []
        for grad in (F, back):
            sigma = ref.solve(grad, True)[0]
            C = ref.stiffness().reshape(-1, 36)
            got.append(torch.cat([sigma, torch.zeros_like(sigma[:, :3]), C], dim=1))
        step = torch.cat([ref.orientation(), ref.orientation(params[:, 5:8])], dim=1)
        return {"there": got[0], "back": got[1], "step": step, "steps": None}
    if call == "stiffness":
        ref.solve(F, True)
        return {"C": ref.stiffness()}
    if call == "cycle":
        there, back = ref.solve(F, True)[0], ref.solve(back, True)[0]
        return {"there": there, "back": back, "u": ref.u}
    sigma, residual = ref.solve(F, False)
    if call == "device":
        return {"sigma": sigma}
    return {"sigma": sigma, "steps": None, "status": None, "residual": residual}
