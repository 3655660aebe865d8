"""Workloads of the engine, as a user's program runs them.

Every case goes through the public Python API: ``LeviathanEngine`` (single
steps and step blocks), ``BatchEngine`` (many networks at once),
``HubTransitions`` (hub-phase transition counts), ``simulate`` (gradients
through a run) and ``DifferentiableReservoir``.  ``listed`` names the cases,
``draw`` makes more of the same ranges, ``prepare`` builds what a program has
in hand before the call, ``run`` makes one pass, ``exact`` gives the pass's
outputs in 64-bit arithmetic and ``work`` its bytes and operations.

Networks are Watts-Strogatz rings (rewired with p = 0.1) with delays uniform
in [1, max_delay], omega ~ N(0, 1), theta ~ U[0, 2 pi) and weights ~ U[0, 1),
the distributions of the benchmark configurations (``graphs.py``).  They are
drawn here with torch.  The graph of a case follows from its sizes and the
state (delays, weights, phases, frequencies) from the seed, as in a study of
one graph from several initial states.
"""

import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from leviathan_v1_b200 import BatchEngine, LeviathanEngine
from leviathan_v1_b200.adjoint import Adjoint, simulate
from leviathan_v1_b200.graphs import Network
from leviathan_v1_b200.hubs import HubTransitions
from leviathan_v1_b200.reservoir import DifferentiableReservoir, make_inputs

DT = 0.05
TWO_PI = 2.0 * math.pi


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # Closed loop on the smallest configuration (N = 1000, k = 20): one
        # step, then the phases are read back -- a controller, a dashboard or
        # a reservoir that looks at every step.
        dict(name="calls_small", kind="calls", N=1000, k=20, max_delay=50, steps=1),
        # The reference's call pattern on a network that fills the GPU: one
        # step() per step of a run, r read after each.
        dict(name="calls_large", kind="calls", N=500_000, k=32, max_delay=64, steps=16),
        # The small plain configuration as it is recorded: 500 steps, r(t),
        # final phases and weights.
        dict(name="run_small", kind="run", N=1000, k=20, max_delay=50, steps=500),
        # The same record of a mid-sized network.
        dict(name="run_mid", kind="run", N=10_000, k=20, max_delay=50, steps=500),
        # The observatory's default size, made odd: ragged last tile.
        dict(name="run_100k", kind="run", N=100_003, k=20, max_delay=50, steps=500),
        # The plain engine at scale: N = 10^6, k = 32, delays up to 64.
        dict(name="run_scale", kind="run", N=1_000_000, k=32, max_delay=64, steps=500),
        # A whole job on that network: engine from host arrays, 20 steps, phases.
        dict(name="job_scale", kind="job", N=1_000_000, k=32, max_delay=64, steps=20),
        # Coupling sweep: networks of uneven size (N log-uniform in
        # [500, 50000], k in {8, 16, 20, 32}), K over [0, 4], controller off,
        # autotuned.
        dict(name="sweep", kind="sweep", nets=128, n_lo=500, n_hi=50_000, max_delay=50,
             steps=40, tuned=True),
        # Ensemble of small networks: the lower end of the sweep's sizes.
        dict(name="sweep_small", kind="sweep", nets=24, n_lo=500, n_hi=2000, max_delay=50,
             steps=200, tuned=False),
        # Transition counts of eight hubs over a run (the front-end of an
        # integrated-information solver).
        dict(name="hubs_mid", kind="hubs", N=10_000, k=20, max_delay=50, steps=200, hubs=8),
        # Gradients of an r(t) loss through a run: omega, weights and K.
        dict(name="adjoint_mid", kind="adjoint", N=10_000, k=20, max_delay=50, steps=200,
             segment=50),
        # One training step of a reservoir: batch of input sequences, readout,
        # gradients of every parameter.
        dict(name="reservoir", kind="reservoir", N=20_000, k=20, max_delay=50, steps=50,
             segment=25, batch=16, n_input=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges (``rng``: random.Random)."""
    kind = rng.choice(["calls", "run", "run", "job", "sweep", "sweep", "hubs", "adjoint",
                       "adjoint", "reservoir"])
    c = dict(kind=kind, k=rng.choice([8, 16, 20, 32]), max_delay=rng.randint(8, 64))
    if kind == "calls":
        c.update(N=_log_int(rng, 500, 500_000), steps=rng.randint(1, 16))
    elif kind == "run":
        N = _log_int(rng, 500, 1_000_000)
        c.update(N=N, steps=_log_int(rng, 16, 500))
    elif kind == "job":
        c.update(N=_log_int(rng, 2000, 1_000_000), steps=rng.randint(5, 20))
    elif kind == "sweep":
        c.pop("k")
        hi = rng.choice([2000, 10_000, 50_000])
        c.update(nets=rng.randint(8, 96), n_lo=500, n_hi=hi, steps=rng.randint(10, 40),
                 tuned=rng.random() < 0.5)
    elif kind == "hubs":
        c.update(N=_log_int(rng, 500, 100_000), steps=rng.randint(20, 200),
                 hubs=rng.randint(2, 10))
    elif kind == "adjoint":
        c.update(N=_log_int(rng, 500, 100_000), k=rng.choice([8, 16, 20]),
                 steps=rng.randint(20, 100), segment=rng.choice([10, 25, 50]))
    else:
        c.update(N=_log_int(rng, 1000, 20_000), k=rng.choice([8, 16, 20]),
                 steps=rng.randint(20, 50), segment=rng.choice([10, 25]),
                 batch=rng.randint(2, 16), n_input=rng.randint(16, 256))
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _network(N, k, max_delay, seed):
    """Watts-Strogatz network of (N, k) as host arrays (symmetric CSR, columns
    sorted, no self-loops or multi-edges), its state drawn from the seed."""
    dev = _device()
    gen = torch.Generator(device=dev).manual_seed(1_000_003 * k + N)
    half = k // 2
    u = torch.arange(N, device=dev).repeat_interleave(half)
    v = (u + torch.arange(1, half + 1, device=dev).repeat(N)) % N
    far = torch.rand(u.numel(), generator=gen, device=dev) < 0.1
    hop = torch.randint(1, N, (u.numel(),), generator=gen, device=dev)
    v = torch.where(far, (u + hop) % N, v)
    und = torch.unique(torch.minimum(u, v) * N + torch.maximum(u, v))
    a, b = und // N, und % N
    key = torch.sort(torch.cat([a * N + b, b * N + a])).values
    row, col = key // N, key % N
    E = key.numel()
    row_ptr = torch.zeros(N + 1, dtype=torch.int64, device=dev)
    row_ptr[1:] = torch.cumsum(torch.bincount(row, minlength=N), 0)
    gen.manual_seed(int(seed))
    delays = torch.randint(1, max_delay + 1, (E,), generator=gen, device=dev)
    weights = torch.rand(E, generator=gen, device=dev)
    theta = torch.rand(N, generator=gen, device=dev) * TWO_PI
    omega = torch.randn(N, generator=gen, device=dev)
    host = lambda t, dt: t.to(dt).cpu().numpy()
    th = host(theta, torch.float32)
    return Network(N, max_delay, host(row_ptr, torch.int32), host(col, torch.int32),
                   host(delays, torch.uint8), host(weights, torch.float32), th, th.copy(),
                   host(omega, torch.float32), meta=dict(k=k))


def _sweep(case, seed):
    """Networks and parameters of a coupling sweep."""
    rng = np.random.default_rng([case["nets"], 77])
    nets, params = [], []
    for b in range(case["nets"]):
        N = int(round(math.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))))
        k = int(rng.choice([8, 16, 20, 32]))
        nets.append(_network(N, k, case["max_delay"], seed * 1009 + b))
        params.append(dict(g=4.0 * b / max(case["nets"] - 1, 1), gain_controller=0))
    return nets, params


def _hub_indices(case, seed):
    rng = np.random.default_rng([int(seed), 78])
    return np.sort(rng.choice(case["N"], case["hubs"], replace=False)).astype(np.int32)


def _target(T, dev, dtype=torch.float32):
    """Target order parameter r*(t) = 0.5 + 0.2 sin(2 pi t / 400)."""
    t = torch.arange(1, T + 1, device=dev, dtype=torch.float64)
    return (0.5 + 0.2 * torch.sin(TWO_PI * t / 400.0)).to(dtype)


def _reservoir_params(case, seed):
    """Input nodes, input weights and readout a trained model would load."""
    rng = np.random.default_rng([int(seed), 79])
    N = case["N"]
    n_in = min(case["n_input"], N)
    nodes = np.sort(rng.choice(N, n_in, replace=False))
    w_in = rng.normal(0.0, 1.0, n_in).astype(np.float32)
    ro = rng.normal(0.0, 1.0 / math.sqrt(2 * N), (2, N)).astype(np.float32)
    x = make_inputs(case["batch"], case["steps"], seed=int(seed))
    return nodes, w_in, ro, x


def prepare(case, seed):
    kind = case["kind"]
    st = dict(kind=kind, case=case)
    if kind == "sweep":
        nets, params = _sweep(case, seed)
        eng = BatchEngine([n.as_dict() for n in nets], params=params)
        if case["tuned"]:
            eng.autotune(DT)
        st.update(eng=eng)
        return st
    net = _network(case["N"], case["k"], case["max_delay"], seed)
    if kind == "job":
        st.update(net=net)
        return st
    if kind == "reservoir":
        nodes, w_in, ro, x = _reservoir_params(case, seed)
        res = DifferentiableReservoir(net, case["batch"], n_input=len(nodes),
                                      T=case["steps"], segment=case["segment"])
        with torch.no_grad():
            res.input_nodes = torch.as_tensor(nodes, device="cuda")
            res.w_in.copy_(torch.as_tensor(w_in))
            res.read_a.copy_(torch.as_tensor(ro[0]))
            res.read_b.copy_(torch.as_tensor(ro[1]))
        st.update(res=res, x=torch.as_tensor(x, device="cuda"))
        return st
    if kind == "adjoint":
        eng = LeviathanEngine(*net.engine_args(), math_mode="accurate")
        adj = Adjoint(eng, segment=case["segment"], max_steps=case["steps"])
        leaf = lambda a: torch.tensor(a, device="cuda", requires_grad=True)
        st.update(eng=eng, adj=adj, omega=leaf(net.omega), w0=leaf(net.weights),
                  K=leaf(np.array([1.5], np.float32)),
                  target=_target(case["steps"], torch.device("cuda")))
        return st
    eng = LeviathanEngine(*net.engine_args())
    if kind == "run" and case["N"] > 200_000:
        eng.autotune(DT)  # long runs at scale tune their variants once
    if kind == "hubs":
        hubs = HubTransitions(_hub_indices(case, seed))
        hubs.attach(eng)
        st.update(hubs=hubs)
    st.update(eng=eng)
    return st


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "calls":
        eng = state["eng"]
        r = np.array([eng.step(DT) for _ in range(case["steps"])], np.float32)
        return r, eng.get_theta()
    if kind == "run":
        eng = state["eng"]
        r = eng.step_n(DT, case["steps"])
        return r, eng.get_theta(), eng.get_weights()
    if kind == "job":
        with LeviathanEngine(*state["net"].engine_args()) as eng:
            r = eng.step_n(DT, case["steps"])
            return r, eng.get_theta()
    if kind == "sweep":
        eng = state["eng"]
        r = eng.step_n(DT, case["steps"])
        return r, eng.get_theta()
    if kind == "hubs":
        r = state["eng"].step_n(DT, case["steps"])
        counts, totals, _, _ = state["hubs"].read()
        return r, counts.astype(np.int64), totals.astype(np.int64)
    if kind == "adjoint":
        omega, w0, K = state["omega"], state["w0"], state["K"]
        for p in (omega, w0, K):
            p.grad = None
        r = simulate(state["adj"], omega, w0, K, case["steps"], DT)
        loss = torch.mean((r[:, 0] - state["target"]) ** 2)
        loss.backward()
        return r.detach(), omega.grad, w0.grad, K.grad
    res = state["res"]
    res.zero_grad(set_to_none=True)
    y, r = res(state["x"], DT)
    loss = res.loss(y, state["x"])
    loss.backward()
    return (y.detach(), r.detach(), res.w_in.grad, res.omega.grad, res.read_a.grad,
            res.read_b.grad, res.read_c.grad)


# ---------------------------------------------------------------------------
# Bytes and operations of one pass
# ---------------------------------------------------------------------------
def _sizes(case):
    """(nodes, edges) stepped at once."""
    if case["kind"] == "sweep":
        # mean of a log-uniform size, mean of k
        m = (case["n_hi"] - case["n_lo"]) / math.log(case["n_hi"] / case["n_lo"])
        nodes = case["nets"] * m
        return nodes, 19.0 * nodes
    copies = case["batch"] if case["kind"] == "reservoir" else 1
    return copies * case["N"], copies * case["N"] * case["k"]


def work(case):
    """A step reads each edge's column, delay, weight and delayed phase and
    writes its weight (17 bytes), and reads or writes 36 bytes per node; about
    40 operations per edge and 80 per node.  A gradient pass is a forward
    step, and a reverse step that reads column, delay, weight and delayed
    phase, reads and writes the weight's adjoint and adds to the source's
    (29 bytes per edge)."""
    n, e = _sizes(case)
    t = case["steps"]
    b, f = 17.0 * e + 36.0 * n, 40.0 * e + 80.0 * n
    if case["kind"] in ("adjoint", "reservoir"):
        b, f = b + 29.0 * e + 72.0 * n, 2.5 * f
    extra = 4.0 * n
    if case["kind"] == "run":
        extra += 4.0 * e
    if case["kind"] == "job":
        extra += 9.0 * e + 16.0 * n
    return {"bytes": b * t + extra, "flops": f * t}


# ---------------------------------------------------------------------------
# The same outputs in 64 bits
# ---------------------------------------------------------------------------
_P = {k: float(np.float32(v)) for k, v in dict(
    eta=0.01, lam=0.001, gamma=0.05, alpha=0.1, kappa_w=0.01, w_min=0.0, w_max=2.0,
    r0=0.5, beta=0.01, mu=0.01, g_rest=1.5, g_min=0.1, g_max=5.0).items()}
_DT = float(np.float32(DT))


class _Model:
    """The model over one or more networks side by side, float64 on torch."""

    def __init__(self, nets, gains, ctrl):
        dev = _device()
        self.dev, self.B, self.ctrl = dev, len(nets), ctrl
        f64 = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)
        i64 = lambda a: torch.as_tensor(np.asarray(a, np.int64), device=dev)
        off = np.cumsum([0] + [n.N for n in nets])
        self.N = int(off[-1])
        self.row = torch.cat([torch.repeat_interleave(torch.arange(n.N, device=dev),
                                                      torch.diff(i64(n.row_ptr))) + int(o)
                              for n, o in zip(nets, off)])
        self.col = torch.cat([i64(n.col_idx) + int(o) for n, o in zip(nets, off)])
        self.d = torch.cat([i64(n.delays) for n in nets])
        self.md = max(n.max_delay for n in nets)
        self.net = torch.cat([torch.full((n.N,), b, device=dev) for b, n in enumerate(nets)])
        self.n_of = f64([n.N for n in nets])
        self.theta = torch.cat([f64(n.theta) for n in nets])
        self.theta_hat = torch.cat([f64(n.theta_hat) for n in nets])
        self.omega = torch.cat([f64(n.omega) for n in nets])
        self.w = torch.cat([f64(n.weights) for n in nets])
        self.g = f64(gains)

    def step(self, ring, t, theta, theta_hat, omega_hat, w, g, omega, drive=None):
        """One step from ring[slot of theta(tau)] = tau mod (max_delay + 1)."""
        diff = theta - theta_hat
        diff = diff - torch.floor(diff / TWO_PI + 0.5) * TWO_PI
        eps = torch.sin(diff)
        theta_hat = theta_hat + _DT * omega_hat
        omega_hat = omega_hat + _P["kappa_w"] * _DT * eps
        bs = self.md + 1
        flat = ring.reshape(-1) if torch.is_tensor(ring) else torch.cat(ring)
        delta = flat[torch.remainder(t - self.d, bs) * self.N + self.col] - theta[self.row]
        delta = delta - torch.floor(delta / TWO_PI + 0.5) * TWO_PI
        S = torch.zeros(self.N, dtype=torch.float64, device=self.dev).index_add(
            0, self.row, w * torch.sin(delta))
        w = w + _DT * (_P["eta"] * torch.cos(delta)
                       * (1.0 - _P["gamma"] * torch.abs(eps)[self.row]) - _P["lam"] * w)
        w = torch.clamp(w, _P["w_min"], _P["w_max"])
        rate = omega + g[self.net] * S - _P["alpha"] * eps
        if drive is not None:
            rate = rate + drive
        x = theta + _DT * rate
        x = x - torch.floor(x / TWO_PI) * TWO_PI
        zero = torch.zeros(self.B, dtype=torch.float64, device=self.dev)
        c = zero.index_add(0, self.net, torch.cos(x)) / self.n_of
        s = zero.index_add(0, self.net, torch.sin(x)) / self.n_of
        r = torch.sqrt(c * c + s * s)
        if self.ctrl:
            g = torch.clamp(g + _DT * (_P["beta"] * (_P["r0"] - r)
                                       - _P["mu"] * (g - _P["g_rest"])),
                            _P["g_min"], _P["g_max"])
        return x, theta_hat, omega_hat, w, g, r

    def run(self, T):
        bs = self.md + 1
        ring = self.theta.repeat(bs, 1)
        s = (self.theta, self.theta_hat, self.omega, self.w, self.g)
        rs = []
        for t in range(T):
            *s, r = self.step(ring, t, *s, self.omega)
            ring[(t + 1) % bs] = s[0]
            rs.append(r)
        return torch.stack(rs), s[0], s[3]

    def run_grad(self, T, omega, w, g, drive=None, readout=None):
        """As ``run`` with autograd; one step's intermediates are kept at a
        time.  drive(t) and readout(theta) are functions of the leaves."""
        bs = self.md + 1
        ring = [self.theta] * bs
        s = (self.theta, self.theta_hat, omega, w, g)
        rs, ys = [], []
        for t in range(T):
            f = lambda *a, t=t: self.step(list(a[:bs]), t, *a[bs:bs + 6],
                                          drive=None if drive is None else drive(t))
            *s, r = checkpoint(f, *ring, *s, omega, use_reentrant=False)
            ring = list(ring)
            ring[(t + 1) % bs] = s[0]
            rs.append(r)
            if readout is not None:
                ys.append(readout(s[0]))
        return torch.stack(rs), (torch.stack(ys) if ys else None)


def exact(case, seed):
    kind, T = case["kind"], case["steps"]
    if kind == "sweep":
        nets, params = _sweep(case, seed)
        m = _Model(nets, [float(np.float32(p["g"])) for p in params], False)
        r, th, _ = m.run(T)
        return r.cpu().numpy(), th.cpu().numpy()
    net = _network(case["N"], case["k"], case["max_delay"], seed)
    if kind == "adjoint":
        m = _Model([net], [1.5], True)
        omega, w0, K = (v.clone().requires_grad_() for v in (m.omega, m.w, m.g))
        r, _ = m.run_grad(T, omega, w0, K)
        torch.mean((r[:, 0] - _target(T, m.dev).double()) ** 2).backward()
        return r.detach(), omega.grad, w0.grad, K.grad
    if kind == "reservoir":
        nodes, w_in, ro, x = _reservoir_params(case, seed)
        B, N = case["batch"], case["N"]
        m = _Model([net] * B, [1.5] * B, True)
        leaf = lambda a: torch.as_tensor(np.asarray(a, np.float64),
                                         device=m.dev).clone().requires_grad_()
        omega, win, ra, rb, rc = (leaf(v) for v in (net.omega, w_in, ro[0], ro[1], [0.0]))
        xd = torch.as_tensor(x, device=m.dev).double()
        idx = torch.as_tensor(nodes, device=m.dev)
        full = torch.zeros(N, dtype=torch.float64, device=m.dev).index_copy(0, idx, win)
        r, y = m.run_grad(
            T, omega.repeat(B), m.w, m.g,
            drive=lambda t: (xd[:, t, None] * full[None, :]).reshape(-1),
            readout=lambda th: (ra * torch.cos(th.view(B, N))
                                + rb * torch.sin(th.view(B, N))).sum(1))
        y, r = y.t() + rc, r.t()
        torch.mean((y[:, :-10] - xd[:, 10:]) ** 2).backward()
        return y.detach(), r.detach(), win.grad, omega.grad, ra.grad, rb.grad, rc.grad
    r, th, w = (v.cpu().numpy() for v in _Model([net], [1.5], True).run(T))
    if kind == "hubs":
        return r[:, 0], None, None  # the counts are whole numbers
    if kind == "run":
        return r[:, 0], th, w
    return r[:, 0], th
