"""The batched geometric step by active items (bitmaps of 128-replica items)
and its paths for rows with many contacts, against the oracle at the sizes
where the layout changes: columns per row around the powers of two and the
32-column slices, rows around 48 and 256 pairs, replicas that return to
susceptible, certain and impossible transitions."""
import numpy as np
import pytest

from replay_b200 import synthetic

pytestmark = pytest.mark.gpu


def _check(oracle, net, n, csr="per-step", **kw):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    g = rb.Graph.from_arrays(net["start"], net["end"], net["u"], net["v"], n)
    sim = rb.Simulation(g, path="batched", csr=csr, transition="geometric", step_size=1800.0, window=1800,
                        start_time=net["t0"], seed=11, ncls_cap=False, **kw)
    okw = {k: int(v) if isinstance(v, bool) else v for k, v in kw.items() if k not in ("M", "iterations")}
    want = oracle.run(net["start"], net["end"], net["u"], net["v"], n, n_replicas=kw["M"], n_steps=kw["iterations"],
                      step_size=1800.0, window=1800, start_time=net["t0"], seed=11, ncls_cap=0, transition=1, **okw)
    np.testing.assert_array_equal(sim.run(), want)


# 1, 2, 3, 5, 9, 17 and 33 columns of 128 replicas: each bitmap layout and a second slice
@pytest.mark.parametrize("replicas", [1, 129, 300, 520, 1030, 2080, 4130])
def test_columns(oracle, replicas):
    net = synthetic.tiny(seed=120, n_nodes=45, n_contacts=900)
    _check(oracle, net, 45, M=replicas, iterations=10, beta=4e-4, p_ei=0.04, p_ir=0.03, p_rs=0.02, initial_count=2)


RULES = [
    dict(p_ei=0.05, p_ir=0.04, initial_count=1),                      # sparse: most items never active
    dict(p_ei=0.05, p_ir=0.04, p_rs=0.3, initial_infected=0.2),       # a rate above 1/16 next to small ones
    dict(p_ei=1.0, p_ir=0.02, initial_infected=0.05),                 # certain E -> I
    dict(p_ir=1.0, has_exposed=False, ir_to_s=True, initial_infected=0.1),  # certain I -> S
    dict(p_ei=0.0, p_ir=0.03, initial_infected=0.1),                  # E never leaves
    dict(p_ir=0.02, has_exposed=False, p_rs=0.01, initial_infected=0.9),    # few susceptibles left
    dict(p_ei=0.0038, p_ir=0.002, p_rs=0.003, initial_infected=0.4),  # every rate below 1/256
]


@pytest.mark.parametrize("rule", range(len(RULES)))
def test_rules(oracle, rule):
    net = synthetic.tiny(seed=121 + rule, n_nodes=70, n_contacts=2500, span=8 * 3600)
    sus = np.random.default_rng(rule).uniform(0, 2, 70).astype(np.float32) if rule % 2 else None
    kw = dict(RULES[rule], **({} if sus is None else {"susceptibility": sus}))
    _check(oracle, net, 70, M=200, iterations=16, beta=3e-4, **kw)


def hubs(degrees, n):
    """A network whose node k meets degrees[k] others in every half hour of two hours."""
    rng = np.random.default_rng(5)
    u, v, s = [], [], []
    for k, deg in enumerate(degrees):
        for w in range(4):
            u.append(np.full(deg, k))
            v.append(len(degrees) + rng.integers(0, n - len(degrees), deg))
            s.append(synthetic.EPOCH_2000 + w * 1800 + rng.integers(0, 1000, deg))
    u, v, s = (np.concatenate(x) for x in (u, v, s))
    e = s + rng.integers(1, 800, len(s))
    return dict(start=s.astype(np.int64), end=e.astype(np.int64), u=u.astype(np.int32), v=v.astype(np.int32),
                t0=synthetic.EPOCH_2000)


@pytest.mark.parametrize("csr", ["per-step", "prebuilt"])
@pytest.mark.parametrize("replicas", [40, 1100, 4200])
def test_rows_with_many_pairs(oracle, replicas, csr):
    n = 1500
    net = hubs([47, 48, 49, 64, 255, 256, 257, 512, 900, 1300], n)
    beta = np.geomspace(1e-8, 3e-3, replicas).astype(np.float32)
    _check(oracle, net, n, csr=csr, M=replicas, iterations=4, beta_per_replica=beta, p_ei=0.3, p_ir=0.05,
           initial_infected=0.05)


def test_row_total_beyond_32_bits(oracle):
    """A row's contact-seconds above 2^32 leave the bit-sliced sums: windows of 2 x 10^8 s."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    rng = np.random.default_rng(3)
    n, w = 60, 200_000_000
    v = np.tile(np.arange(1, n), 2).astype(np.int32)
    s = synthetic.EPOCH_2000 + rng.integers(0, 1000, len(v))
    e = s + w + rng.integers(0, 1000, len(v))
    u = np.zeros(len(v), np.int32)
    kw = dict(step_size=float(w), window=w, start_time=synthetic.EPOCH_2000, seed=4, beta=3e-10, p_ei=0.3, p_ir=0.1,
              initial_infected=0.3)
    g = rb.Graph.from_arrays(s, e, u, v, n)
    sim = rb.Simulation(g, M=150, iterations=3, path="batched", transition="geometric", ncls_cap=False, **kw)
    want = oracle.run(s, e, u, v, n, n_replicas=150, n_steps=3, transition=1, ncls_cap=0, **kw)
    assert (want[1:, :, 0] > 0).any()
    np.testing.assert_array_equal(sim.run(), want)
