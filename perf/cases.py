"""The work a user has this library do, as cases that can be timed: whole
calls through the public Python API over seeded synthetic networks with the
shapes and distributions of the configurations in replay_b200/synthetic.py
and bench.py.

A case's "kind" selects the call:
  replay     Simulation.run() of a geometric replay on one network
  batch      Simulation.run() of many independent networks in one replay
  dense      Simulation.run() on a power-law contact network (hub rows)
  countdown  Simulation.run() under the countdown rule (the `replay` default)
  end2end    Graph.from_arrays + Simulation + run + close on host arrays
  text       Simulation.run_text(): node-state CSV lines of every step
  meanfield  expected-value replay: forward and gradients of a daily-incidence fit

Monte Carlo outputs are whole numbers (counts, text bytes) and have no value
outside the library's random streams; the mean-field cases have one in 64
bits (`exact`).
"""
import math

import numpy as np
import torch

import replay_b200
from replay_b200.meanfield import MeanField, daily_incidence

T0 = 946684800  # 2000-01-01T00:00:00Z
DAY = 86400


def listed():
    return [
        # a small study's quick look: a few hundred people, two days, few replicas (latency and launches)
        dict(name="replay_smallest", kind="replay", nodes=300, contacts=9_000, steps=48, step=3600, replicas=128,
             median=600, sigma=1.0, beta=6e-5, csr="per-step"),
        # the small SEIR configuration: one community, a week, 1,000 replicas
        dict(name="replay_small", kind="replay", nodes=1_000, contacts=50_000, steps=168, step=3600, replicas=1_000,
             median=600, sigma=1.0, beta=2e-5, csr="per-step"),
        # a town with odd sizes, waning immunity, per-node susceptibility, Bernoulli seeding, and windows kept
        # for many replays (csr="prebuilt")
        dict(name="replay_town_waning", kind="replay", nodes=20_011, contacts=2_000_000, steps=168, step=3600,
             replicas=1_001, median=900, sigma=1.2, beta=3e-5, p_rs=1 / 240, susceptibility=True,
             initial=0.002, csr="prebuilt"),
        # the replica sweep, the headline configuration: 64 betas x 64 seeds on 100 communities, two weeks
        dict(name="replay_sweep", kind="replay", nodes=100_000, contacts=20_000_000, steps=336, step=3600,
             replicas=4_096, median=900, sigma=1.2, betas=64, communities=100, daily=True, csr="per-step"),
        # the uneven batch: 256 networks of 500..50,000 nodes in one replay, sparse half-hour windows (ten of
        # its thirty days)
        dict(name="batch_uneven", kind="batch", networks=256, smallest=500, largest=50_000, contacts_per_node=20 / 3,
             steps=480, step=1800, replicas=128, median=300, sigma=1.0, beta=3e-5),
        # the dense stress network, SIR with 16,384 replicas and hub rows of thousands of contacts (three of
        # its thirty days)
        dict(name="dense_hubs", kind="dense", nodes=5_000, contacts=5_000_000, steps=288, step=900, replicas=16_384,
             mean=1200, beta=1e-5, initial=5),
        # the reference's own benchmark scenario "villages" (population 1,000, 10,000 replicas, countdown rule)
        dict(name="countdown_villages", kind="countdown", nodes=1_000, groups=100, inner=0.9, inter=0.05, steps=100,
             step=3600, replicas=10_000, initial=0.5, infect_prob=1.0, exposed=3600, infectious=3600, resistant=0),
        # a small study under the countdown rule: 5,000 nodes, long durations, 64 replicas
        dict(name="countdown_study", kind="countdown", nodes=5_000, contacts=904_000, communities=5, steps=336, step=3600,
             median=900, sigma=1.2, replicas=64, initial=0.004, infect_prob=0.0773, exposed=172_800,
             infectious=432_000, resistant=100_000_000),
        # a user's whole job on new contact data: upload, index, plan, replay, counts
        dict(name="end2end_sweep", kind="end2end", nodes=100_000, contacts=20_000_000, steps=336, step=3600,
             replicas=4_096, median=900, sigma=1.2, betas=64, communities=100, daily=True, csr="per-step"),
        # --node-state-out of a small replay: every replica's node states as CSV lines
        dict(name="text_small", kind="text", nodes=1_000, contacts=7_000, steps=24, step=3600, replicas=64,
             median=600, sigma=1.0, beta=2e-5, csr="per-step"),
        # one iteration of a calibration on the sweep's network, and on its first two communities
        dict(name="meanfield_sweep", kind="meanfield", nodes=100_000, contacts=20_000_000, steps=336, step=3600,
             median=900, sigma=1.2, beta=3e-5, communities=100, daily=True),
        dict(name="meanfield_small", kind="meanfield", nodes=2_000, contacts=360_000, steps=336, step=3600,
             median=900, sigma=1.2, beta=3e-5, communities=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["replay", "replay", "batch", "dense", "countdown", "countdown", "end2end", "text", "meanfield"])
    c = dict(kind=kind)
    if kind in ("replay", "end2end"):
        n = _log(rng, 200, 100_000)
        steps = _log(rng, 24, 336)
        m = _log(rng, 16, max(16, min(4_096, 40_000_000_000 // (n * steps))))
        c.update(nodes=n, contacts=min(8_000_000, n * _log(rng, 10, 200)), steps=steps, step=rng.choice([900, 1800, 3600]),
                 replicas=m, median=rng.choice([300, 600, 900]), sigma=rng.choice([1.0, 1.2]),
                 beta=math.exp(rng.uniform(math.log(1e-5), math.log(1e-4))), csr=rng.choice(["per-step", "prebuilt"]))
        if rng.random() < 0.3:
            c.update(betas=rng.choice([4, 16, 64]))
        if rng.random() < 0.3:
            c.update(p_rs=1 / rng.choice([120, 240]))
        if rng.random() < 0.3:
            c.update(susceptibility=True)
        if rng.random() < 0.3:
            c.update(initial=rng.choice([0.001, 0.01]))
        rule = rng.random()
        if rule < 0.15:
            c.update(exposed=False)  # SIR
        elif rule < 0.25:
            c.update(exposed=False, ir_to_s=True)  # SIS
    elif kind == "batch":
        c.update(networks=_log(rng, 4, 256), smallest=rng.choice([100, 500]), largest=_log(rng, 1_000, 30_000),
                 contacts_per_node=rng.uniform(3, 20), steps=_log(rng, 48, 400), step=rng.choice([900, 1800, 3600]),
                 replicas=_log(rng, 16, 200), median=300, sigma=1.0, beta=rng.choice([1e-5, 3e-5, 1e-4]))
    elif kind == "dense":
        n = _log(rng, 500, 5_000)
        c.update(nodes=n, contacts=_log(rng, 100_000, 4_000_000), steps=_log(rng, 48, 250), step=900,
                 replicas=_log(rng, 100, 16_384), mean=1200, beta=rng.choice([3e-6, 1e-5]), initial=5)
    elif kind == "countdown":
        n = _log(rng, 200, 20_000)
        steps = _log(rng, 24, 200)
        c.update(nodes=n, contacts=n * _log(rng, 10, 100), communities=1, steps=steps, step=3600, median=900, sigma=1.2,
                 replicas=_log(rng, 16, max(16, min(10_000, 600_000_000 // (n * steps)))), initial=rng.choice([0.004, 0.05]),
                 infect_prob=rng.uniform(0.02, 0.3), exposed=3600 * rng.randint(1, 60),
                 infectious=3600 * rng.randint(1, 120), resistant=rng.choice([0, 36_000, 100_000_000]))
    elif kind == "text":
        c.update(nodes=_log(rng, 100, 1_500), contacts=_log(rng, 2_000, 10_000), steps=rng.randint(6, 40), step=3600,
                 replicas=_log(rng, 8, 64), median=600, sigma=1.0, beta=2e-5, csr="per-step")
    else:
        n = _log(rng, 500, 60_000)
        c.update(nodes=n, contacts=min(6_000_000, n * _log(rng, 10, 180)), steps=24 * rng.randint(1, 14), step=3600,
                 median=900, sigma=1.2, beta=rng.choice([1e-5, 3e-5]), communities=1)
    return c


# ---------------------------------------------------------------------------
# Networks (made on the GPU, handed to the library as host arrays)


def _uniform_pairs(n, size, base, g):
    """n distinct pairs inside [base, base + size) (tensors or numbers)."""
    a = (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * size).long()
    b = (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (size - 1)).long()
    b = b + (b >= a)
    return torch.minimum(a, b) + base, torch.maximum(a, b) + base


def _lognormal(n, c, g):
    z = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    return torch.clamp(torch.round(torch.exp(math.log(c["median"]) + c["sigma"] * z)), 1, 8 * 3600).long()


def _starts(n, span, daily, g):
    if not daily:
        return T0 + (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * span).long()
    got = []  # uniform candidates thinned by the daily rate 1 + 0.8 sin(2 pi t / 24 h)
    while sum(len(x) for x in got) < n:
        t = (torch.rand(2 * n, generator=g, device="cuda", dtype=torch.float64) * span).long()
        keep = torch.rand(2 * n, generator=g, device="cuda", dtype=torch.float64) * 1.8
        got.append(t[keep < 1.0 + 0.8 * torch.sin(2 * math.pi * t.double() / DAY)])
    return T0 + torch.cat(got)[:n]


def _contacts(c, seed):
    """(start, end, u, v, n_nodes, network offsets or None), GPU tensors but the offsets."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    span = c["steps"] * c["step"]
    offsets = None
    if c["kind"] == "batch":
        rng = np.random.default_rng(int(seed))
        sizes = np.rint(np.exp(rng.uniform(np.log(c["smallest"]), np.log(c["largest"]), c["networks"]))).astype(np.int64)
        offsets = np.concatenate([[0], np.cumsum(sizes)])
        per = np.rint(sizes * c["contacts_per_node"]).astype(np.int64)
        n, nodes = int(per.sum()), int(offsets[-1])
        per = torch.from_numpy(per).cuda()
        u, v = _uniform_pairs(n, torch.repeat_interleave(torch.from_numpy(sizes).cuda(), per),
                              torch.repeat_interleave(torch.from_numpy(offsets[:-1]).cuda(), per), g)
        start = _starts(n, span, False, g)
        end = start + _lognormal(n, c, g)
        offsets = offsets.astype(np.int32)
    elif c["kind"] == "dense":
        n, nodes = c["contacts"], c["nodes"]
        activity = (1 - torch.rand(nodes, generator=g, device="cuda", dtype=torch.float64)) ** (-1 / 1.2)
        cdf = torch.cumsum(activity / activity.sum(), 0)
        cdf[-1] = 1.0
        a = torch.searchsorted(cdf, torch.rand(n, generator=g, device="cuda", dtype=torch.float64))
        b = torch.searchsorted(cdf, torch.rand(n, generator=g, device="cuda", dtype=torch.float64))
        b = torch.where(a == b, (a + 1) % nodes, b)
        u, v = torch.minimum(a, b), torch.maximum(a, b)
        start = _starts(n, span, False, g)
        x = -c["mean"] * torch.log1p(-torch.rand(n, generator=g, device="cuda", dtype=torch.float64))
        end = start + torch.clamp(torch.round(x), 1, 12 * 3600).long()
    elif "groups" in c:  # the group model: each step, pairs of one group meet with prob inner, others with inter
        nodes = c["nodes"]
        i, j = torch.triu_indices(nodes, nodes, 1, device="cuda")
        p = torch.where(i % c["groups"] == j % c["groups"], c["inner"], c["inter"])
        k, u, v = [], [], []
        for t in range(c["steps"]):
            at = torch.nonzero(torch.rand(len(p), generator=g, device="cuda") < p).reshape(-1)
            k.append(torch.full_like(at, T0 + t * c["step"]))
            u.append(i[at])
            v.append(j[at])
        k, u, v = torch.cat(k), torch.cat(u), torch.cat(v)
        a = (torch.rand(len(k), generator=g, device="cuda", dtype=torch.float64) * c["step"]).long()
        b = (torch.rand(len(k), generator=g, device="cuda", dtype=torch.float64) * c["step"]).long()
        start, end = k + torch.minimum(a, b), k + torch.maximum(a, b)
    else:
        n, nodes = c["contacts"], c["nodes"]
        comm = c.get("communities", 1)
        size = nodes // comm
        inside = n if comm == 1 else round(0.9 * n)
        base = (torch.rand(inside, generator=g, device="cuda", dtype=torch.float64) * comm).long() * size
        u, v = _uniform_pairs(inside, size, base, g)
        if inside < n:
            a, b = _uniform_pairs(n - inside, nodes, 0, g)
            u, v = torch.cat([u, a]), torch.cat([v, b])
        start = _starts(n, span, c.get("daily", False), g)
        end = start + _lognormal(n, c, g)
    return start, end, u, v, nodes, offsets


def _host(c, seed):
    start, end, u, v, nodes, offsets = _contacts(c, seed)
    return (start.cpu().numpy(), end.cpu().numpy(), u.int().cpu().numpy(), v.int().cpu().numpy(), nodes), offsets


def _params(c, seed, nodes):
    p = dict(M=c["replicas"], iterations=c["steps"], step_size=float(c["step"]), window=c["step"], start_time=T0,
             seed=int(seed) + 1)
    if c["kind"] == "countdown":
        p.update(transition="countdown", initial_infected=c["initial"], infect_prob=c["infect_prob"],
                 exposed_duration=c["exposed"], infectious_duration=c["infectious"], resistant_duration=c["resistant"])
        return p
    per_hour = c["step"] / 3600
    p.update(transition="geometric", p_ir=per_hour / 120, p_rs=per_hour * c.get("p_rs", 0.0))
    if c["kind"] == "dense" or not c.get("exposed", True):
        p.update(has_exposed=False, p_ir=per_hour / 72, ir_to_s=c.get("ir_to_s", False))
    else:
        p.update(p_ei=per_hour / 48)
    if "betas" in c:
        beta = np.logspace(math.log10(5e-6), -4, c["betas"])
        p.update(beta_per_replica=np.sort(np.resize(beta, c["replicas"])).astype(np.float32))
    else:
        p.update(beta=c["beta"])
    if isinstance(c.get("initial"), float):
        p.update(initial_infected=c["initial"])
    else:
        p.update(initial_count=c.get("initial", 20 if nodes >= 20_000 else 10))
    if c.get("susceptibility"):
        p.update(susceptibility=np.random.default_rng(int(seed)).uniform(0.5, 1.5, nodes).astype(np.float32))
    if "csr" in c:
        p.update(csr=c["csr"])
    return p


# ---------------------------------------------------------------------------


class _Fit:
    """A calibration's objects: the mean-field replay, its inputs and target."""

    def __init__(self, c, seed):
        arrays, _ = _host(c, seed)
        self.graph = replay_b200.Graph.from_arrays(*arrays)
        self.mf = MeanField(self.graph, iterations=c["steps"], step_size=float(c["step"]), window=c["step"], start_time=T0)
        self.x0, self.sus, self.target = _fit_inputs(c, seed)
        self.x0.requires_grad_()
        self.sus.requires_grad_()
        self.beta, self.p_ei, self.p_ir = (torch.tensor(x, device="cuda", requires_grad=True)
                                           for x in (c["beta"], 1 / 48, 1 / 120))

    def __del__(self):
        if hasattr(self, "mf"):
            self.mf.close()


def _fit_inputs(c, seed):
    n, days = c["nodes"], c["steps"] // 24
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 7)
    x0 = torch.zeros(4, n, device="cuda")
    x0[2] = 2e-4 * (0.5 + torch.rand(n, generator=g, device="cuda"))
    x0[0] = 1 - x0[2]
    sus = 0.5 + torch.rand(n, generator=g, device="cuda")
    target = n * 4e-4 * (1 + 0.2 * torch.arange(days, device="cuda"))
    return x0, sus, target


def prepare(case, seed):
    c = case
    if c["kind"] == "meanfield":
        return _Fit(c, seed)
    arrays, offsets = _host(c, seed)
    p = _params(c, seed, arrays[4])
    if c["kind"] == "end2end":
        return dict(kind="end2end", arrays=arrays, params=p)
    graph = replay_b200.Graph.from_arrays(*arrays)
    text = None
    if c["kind"] == "text":
        p.update(record_node_states=True)
        # a buffer for every step's lines, of at most 34 characters each here
        text = np.zeros((c["steps"] + 1, 34 * c["nodes"] * c["replicas"]), np.uint8)
    sim = replay_b200.Simulation(graph, networks=offsets, **p)
    return dict(kind=c["kind"], graph=graph, sim=sim, text=text)


def run(state):
    if isinstance(state, _Fit):
        s = state
        incidence, final = s.mf(s.x0, s.beta, susceptibility=s.sus, p_ei=s.p_ei, p_ir=s.p_ir)
        loss = ((daily_incidence(incidence, 24) - s.target) ** 2).mean()
        gx0, gsus, gbeta, gei, gir = torch.autograd.grad(loss, [s.x0, s.sus, s.beta, s.p_ei, s.p_ir])
        return dict(incidence=incidence, final=final, loss=loss, grad_x0=gx0, grad_sus=gsus, grad_beta=gbeta,
                    grad_p_ei=gei, grad_p_ir=gir)
    if state["kind"] == "end2end":
        graph = replay_b200.Graph.from_arrays(*state["arrays"])
        sim = replay_b200.Simulation(graph, **state["params"])
        counts = sim.run()
        sim.close()
        graph.close()
        return counts
    if state["kind"] == "text":
        text, filled = state["text"], [0] * len(state["text"])

        def write(step, timestamp, data):
            at = filled[step]
            text[step, at:at + len(data)] = np.frombuffer(data, np.uint8)
            filled[step] = at + len(data)

        counts = state["sim"].run_text(write)
        return dict(counts=counts, text=text)
    return state["sim"].run()


def work(case):
    """Contacts read once and results written once (the state between steps
    is the library's own); the mean-field's products count as operations."""
    c = case
    if c["kind"] == "batch":
        span = math.log(c["largest"] / c["smallest"])
        contacts = c["networks"] * (c["largest"] - c["smallest"]) / span * c["contacts_per_node"]
    elif "groups" in c:
        n, k = c["nodes"], c["nodes"] / c["groups"]
        inner = n * (k - 1) / 2
        contacts = c["steps"] * (inner * c["inner"] + (n * (n - 1) / 2 - inner) * c["inter"])
    else:
        contacts = c["contacts"]
    if c["kind"] == "meanfield":
        # forward and adjoint: two multiply-adds per contact and direction each, at least
        return dict(bytes=24 * contacts + 4 * (9 + 4) * c["nodes"], flops=8 * contacts)
    out = (c["steps"] + 1) * c["replicas"] * 16 * c.get("networks", 1)
    if c["kind"] == "text":
        out += (c["steps"] + 1) * c["replicas"] * c["nodes"] * 30
    return dict(bytes=24 * contacts + out, flops=0)


def exact(case, seed):
    c = case
    if c["kind"] != "meanfield":
        return None
    start, end, u, v, n, _ = _contacts(c, seed)
    step, steps = c["step"], c["steps"]
    # one entry per (contact, window it overlaps), ordered by window
    first = (start - T0) // step
    last = torch.clamp((end - 1 - T0) // step, max=steps - 1)
    reps = torch.clamp(last - first + 1, min=0)
    k = torch.repeat_interleave(torch.arange(len(start), device="cuda"), reps)
    win = first[k] + torch.arange(len(k), device="cuda") - torch.repeat_interleave(torch.cumsum(reps, 0) - reps, reps)
    ws = T0 + win * step
    weight = (torch.minimum(end[k], ws + step) - torch.maximum(start[k], ws)).double()
    win, order = torch.sort(win)
    a, b, weight = u[k][order], v[k][order], weight[order]
    cut = torch.searchsorted(win, torch.arange(steps + 1, device="cuda")).tolist()
    x0, sus, target = (t.double() for t in _fit_inputs(c, seed))
    rates = [torch.tensor(x, device="cuda").double() for x in (c["beta"], 1 / 48, 1 / 120)]
    beta, p_ei, p_ir = rates
    leaves = [x0, sus, beta, p_ei, p_ir]
    for t in leaves:
        t.requires_grad_()
    S, E, I, R = x0
    incidence = []
    for t in range(steps):
        i, j, w = a[cut[t]:cut[t + 1]], b[cut[t]:cut[t + 1]], weight[cut[t]:cut[t + 1]]
        e = torch.zeros_like(I).index_add(0, i, w * I[j]).index_add(0, j, w * I[i])
        new = S * -torch.expm1(-beta * sus * e)
        incidence.append(new.sum())
        S, E, I, R = S - new, E * (1 - p_ei) + new, I * (1 - p_ir) + p_ei * E, R + p_ir * I
    incidence = torch.stack(incidence)
    loss = ((daily_incidence(incidence, 24) - target) ** 2).mean()
    gx0, gsus, gbeta, gei, gir = torch.autograd.grad(loss, leaves)
    return dict(incidence=incidence.detach(), final=torch.stack([S, E, I, R]).detach(), loss=loss.detach(), grad_x0=gx0,
                grad_sus=gsus, grad_beta=gbeta, grad_p_ei=gei, grad_p_ir=gir)
