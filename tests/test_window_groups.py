"""Windows built in groups (one chain of launches for many consecutive
windows): per-step replays against the oracle where the grouping has edges."""
import numpy as np
import pytest

from replay_b200 import synthetic

CASES = [
    # 700 windows of a tiny network: more than one full group of 256, a remainder, empty windows at the end
    dict(n=20, contacts=900, span=550 * 300, steps=700, step=300, kw=dict(transition="geometric", beta=1e-3, p_ei=0.2, p_ir=0.1)),
    # the hit cap binds in some windows of a group and not in others
    dict(n=30, contacts=400, span=6 * 3600, steps=24, step=900, cap=True,
         kw=dict(transition="countdown", infect_prob=0.4, exposed_duration=900, infectious_duration=2700,
                 resistant_duration=900)),
    # several scan tiles per window, FP32 rows sorted in a group, two steps per window
    dict(n=9000, contacts=40_000, span=6 * 3600, steps=12, step=1800, window=3600,
         kw=dict(transition="countdown", infect_prob=0.4, exposed_duration=900, infectious_duration=7200,
                 resistant_duration=900)),
]


def capped(net, c):
    """Contacts whose sublist count (the reference's hit cap) is small: one long
    contact over non-nested ones of one duration, every 16th of which holds another."""
    k = np.arange(c["contacts"])
    start = net["t0"] + k * (c["span"] // c["contacts"])
    start[0], start[1::16] = net["t0"], start[:-1:16] + 1
    end = start + 1200
    end[0], end[1::16] = net["t0"] + c["span"] + 1300, start[1::16] + 60
    return dict(net, start=start, end=end)


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(CASES)))
def test_grouped_windows_match_oracle(oracle, case):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    c = CASES[case]
    net = synthetic.tiny(seed=90 + case, n_nodes=c["n"], n_contacts=c["contacts"], span=c["span"], max_dur=3000)
    if c.get("cap"):
        net = capped(net, c)
    kw = dict(step_size=float(c["step"]), window=c.get("window", c["step"]), start_time=net["t0"], seed=5,
              ncls_cap=int(bool(c.get("cap"))), initial_infected=0.1)
    g = rb.Graph.from_arrays(net["start"], net["end"], net["u"], net["v"], c["n"])
    sim = rb.Simulation(g, M=40, iterations=c["steps"], path="batched", csr="per-step", **kw, **c["kw"])
    mode = 0 if c["kw"]["transition"] == "countdown" else 1
    want = oracle.run(net["start"], net["end"], net["u"], net["v"], c["n"], n_replicas=40, n_steps=c["steps"],
                      **kw, **dict(c["kw"], transition=mode))
    np.testing.assert_array_equal(sim.run(), want)
    np.testing.assert_array_equal(sim.run(), want)  # the workspaces are reused


# fewer than one row in eight with a contact per window: windows that list their rows, alone and in a batch,
# with a hub row above 48 and above 256 pairs, windows without contacts, two steps per window
@pytest.mark.gpu
@pytest.mark.parametrize("nodes,hub,window,networks", [(5000, 0, 900, 1), (9000, 60, 900, 3), (40_000, 700, 1800, 1)])
def test_sparse_windows_match_oracle(oracle, nodes, hub, window, networks):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    rng = np.random.default_rng(hub)
    first = np.array([0, nodes // 3, nodes // 2, nodes][:networks] + [nodes], np.int32)
    t0, m = synthetic.EPOCH_2000, 4 * nodes // 10
    start = t0 + rng.integers(0, 20 * 900, m)
    net = rng.integers(0, networks, m)
    lo, hi = first[net].astype(np.int64), first[net + 1].astype(np.int64)
    u = (lo + rng.integers(0, 1 << 30, m) % (hi - lo - 1)).astype(np.int32)
    v = (u + 1).astype(np.int32)
    if hub:  # node 3 meets `hub` others in one window
        start = np.concatenate([start, np.full(hub, t0 + 5 * 900 + 10)])
        u = np.concatenate([u, np.full(hub, 3, np.int32)])
        v = np.concatenate([v, 10 + np.arange(hub, dtype=np.int32)])
    end = start + rng.integers(1, 800, len(start))
    kw = dict(step_size=900.0, window=window, start_time=t0, seed=3, ncls_cap=0, beta=2e-3, p_ei=0.2, p_ir=0.05,
              initial_infected=0.2)
    g = rb.Graph.from_arrays(start, end, u, v, nodes)
    batch = {"networks": first} if networks > 1 else {}
    sim = rb.Simulation(g, M=70, iterations=24, transition="geometric", path="batched", csr="per-step", **batch, **kw)
    if networks > 1:
        batch = {"net_first": first}
    want = oracle.run(start, end, u, v, nodes, n_replicas=70, n_steps=24, transition=1, **batch, **kw)
    np.testing.assert_array_equal(sim.run(), want)
    np.testing.assert_array_equal(sim.run(), want)


# prebuilt windows: grouped, empty ones among them, several windows' lists of heavy rows in one arena
@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(CASES)))
def test_prebuilt_windows_match_oracle(oracle, case):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    c = CASES[case]
    net = synthetic.tiny(seed=70 + case, n_nodes=c["n"], n_contacts=c["contacts"], span=c["span"], max_dur=3000)
    if c.get("cap"):
        net = capped(net, c)
    net["u"][::3] = 0  # a hub
    net["v"][::3] = 1 + net["v"][::3] % (c["n"] - 1)
    kw = dict(step_size=float(c["step"]), window=c.get("window", c["step"]), start_time=net["t0"], seed=5,
              ncls_cap=int(bool(c.get("cap"))), initial_infected=0.1)
    g = rb.Graph.from_arrays(net["start"], net["end"], net["u"], net["v"], c["n"])
    sim = rb.Simulation(g, M=40, iterations=c["steps"], path="batched", csr="prebuilt", **kw, **c["kw"])
    mode = 0 if c["kw"]["transition"] == "countdown" else 1
    want = oracle.run(net["start"], net["end"], net["u"], net["v"], c["n"], n_replicas=40, n_steps=c["steps"],
                      **kw, **dict(c["kw"], transition=mode))
    np.testing.assert_array_equal(sim.run(), want)


# candidates for more than 1 GB of pairs: the arena is sized by a first pass over the windows
@pytest.mark.gpu
def test_prebuilt_arena_sized_by_a_first_pass():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    rng = np.random.default_rng(8)
    n, m, t0 = 2000, 3_000_000, synthetic.EPOCH_2000
    start = t0 - m + np.arange(m)
    end = start + m + 86_400 + 3600
    u = rng.integers(0, n, m).astype(np.int32)
    v = ((u + rng.integers(1, n, m)) % n).astype(np.int32)
    kw = dict(M=32, iterations=24, step_size=3600.0, window=3600, start_time=t0, seed=4, ncls_cap=0, beta=1e-8,
              p_ei=0.2, p_ir=0.1, initial_infected=0.1, transition="geometric", path="batched")
    g = rb.Graph.from_arrays(start, end, u, v, n)
    runs = {}
    for csr in ("per-step", "prebuilt"):
        sim = rb.Simulation(g, csr=csr, **kw)
        runs[csr] = sim.run()
        nnz = sim.info["nnz_total"]
    pairs = len(np.unique(np.minimum(u, v).astype(np.int64) * n + np.maximum(u, v)))
    assert nnz == 24 * 2 * pairs  # every contact spans every window
    np.testing.assert_array_equal(runs["prebuilt"], runs["per-step"])
    assert runs["prebuilt"][-1, :, 3].max() < n
