"""The batched countdown rule as sets of replicas that change at fixed ages,
against the oracle where its layout and its counters change: rows of fewer and
more than 32 words, several changed rows per warp (vertical counters), rows of
more than 32 pairs, durations that skip classes, certain infections; and
against the code table, which takes replays too large for the sets."""
import numpy as np
import pytest

from replay_b200 import synthetic

pytestmark = pytest.mark.gpu

RULES = [
    dict(initial_infected=0.3, infect_prob=0.3, exposed_duration=3600, infectious_duration=7200, resistant_duration=1800),
    dict(initial_infected=0.5, infect_prob=1.0, exposed_duration=1800, infectious_duration=1800, resistant_duration=0),
    dict(initial_count=3, infect_prob=0.6, exposed_duration=0, infectious_duration=5000, resistant_duration=100000000),
    dict(initial_infected=0.1, infect_prob=0.2, exposed_duration=2500, infectious_duration=0, resistant_duration=3600),
    dict(initial_infected=0.2, infect_prob=0.0, exposed_duration=1800, infectious_duration=3600, resistant_duration=0),
]


def _rb():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200
    return replay_b200


@pytest.mark.parametrize("rule", range(len(RULES)))
@pytest.mark.parametrize("replicas,contacts", [(33, 2000), (500, 4000), (1100, 4000)])
def test_sets_match_oracle(oracle, rule, replicas, contacts):
    rb = _rb()
    n = 71
    net = synthetic.tiny(seed=130 + rule, n_nodes=n, n_contacts=contacts, span=8 * 3600)
    kw = dict(step_size=1800.0, window=3600, start_time=net["t0"], seed=8, **RULES[rule])
    g = rb.Graph.from_arrays(net["start"], net["end"], net["u"], net["v"], n)
    sim = rb.Simulation(g, M=replicas, iterations=14, path="batched", **kw)
    want = oracle.run(net["start"], net["end"], net["u"], net["v"], n, n_replicas=replicas, n_steps=14,
                      transition=0, **kw)
    np.testing.assert_array_equal(sim.run(), want)
    np.testing.assert_array_equal(sim.run(), want)


def test_node_states_follow_the_counts():
    rb = _rb()
    net = synthetic.tiny(seed=140, n_nodes=50, n_contacts=2000, span=8 * 3600)
    g = rb.Graph.from_arrays(net["start"], net["end"], net["u"], net["v"], 50)
    sim = rb.Simulation(g, M=70, iterations=12, path="batched", record_node_states=True, step_size=1800.0, window=1800,
                        start_time=net["t0"], **RULES[0])
    seen = []
    counts = sim.run(lambda k, ts, states: seen.append(states) and None)
    for k, states in enumerate(seen):
        got = np.stack([(states == c).sum(axis=1) for c in (1, 2, 3, 0)], axis=1)
        np.testing.assert_array_equal(got, counts[k])


def test_code_table_gives_the_same_counts():
    """200,000 nodes x 4,096 replicas x 170 ages are more sets than are kept;
    the first replicas alone are not."""
    rb = _rb()
    n, T = 200_000, 172
    rng = np.random.default_rng(9)
    m = 400_000
    u = rng.integers(0, n - 1, m).astype(np.int32)
    v = (u + 1 + rng.integers(0, 50, m) % (n - u - 1)).astype(np.int32)
    s = synthetic.EPOCH_2000 + rng.integers(0, T * 3600, m)
    e = s + rng.integers(600, 7200, m)
    g = rb.Graph.from_arrays(s, e, u, v, n)
    kw = dict(iterations=T, step_size=3600.0, window=3600, start_time=synthetic.EPOCH_2000, path="batched", seed=6,
              initial_infected=0.02, infect_prob=0.3, exposed_duration=172_800, infectious_duration=432_000,
              resistant_duration=100_000_000)
    small = rb.Simulation(g, M=64, **kw)
    want = small.run()
    small.close()
    big = rb.Simulation(g, M=4096, **kw)
    assert big.info["device_bytes"] < 8 << 30  # codes, not 170 sets of 102 MB
    np.testing.assert_array_equal(big.run()[:, :64], want)
