"""The countdown rule by the code table (replays too large for the sets of
replicas), against the oracle: tables of one and two bytes, replicas that do
not fill a word, several words and slices, several networks, node states.
rp_sim_create_bounded creates the simulations, without room for the sets."""
import ctypes as C

import numpy as np
import pytest

from replay_b200 import synthetic
from test_countdown_sets import RULES
from test_gpu_parity import COUNTDOWN_CASES, _oracle_kw

pytestmark = pytest.mark.gpu


@pytest.fixture
def codes(monkeypatch):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    L = rb.lib()
    create = L.rp_sim_create_bounded
    create.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int32, C.c_int64, C.c_void_p]
    create.restype = C.c_int
    monkeypatch.setattr(L, "rp_sim_create", lambda g, p, out: create(g, p, None, 1, 0, out))
    monkeypatch.setattr(L, "rp_sim_create_batch", lambda g, p, first, n, out: create(g, p, first, n, 0, out))
    return rb


def _graph(rb, net):
    return rb.Graph.from_arrays(net["start"], net["end"], net["u"], net["v"], net["n_nodes"])


@pytest.mark.parametrize("case", range(len(COUNTDOWN_CASES)))
@pytest.mark.parametrize("csr", ["per-step", "prebuilt"])
def test_parity_cases(codes, oracle, case, csr):
    net = synthetic.tiny(seed=10 + case, n_nodes=50, n_contacts=800)
    kw = dict(COUNTDOWN_CASES[case], start_time=net["t0"], seed=99 + case, transition="countdown")
    sim = codes.Simulation(_graph(codes, net), path="batched", csr=csr, **kw)
    want = oracle.run(net["start"], net["end"], net["u"], net["v"], net["n_nodes"], **_oracle_kw(kw))
    np.testing.assert_array_equal(sim.run(), want)
    np.testing.assert_array_equal(sim.run(), want)


@pytest.mark.parametrize("rule", range(len(RULES)))
@pytest.mark.parametrize("replicas", [1, 33, 500, 1100, 4130])
def test_replicas(codes, oracle, rule, replicas):
    net = synthetic.tiny(seed=130 + rule, n_nodes=71, n_contacts=3000, span=8 * 3600)
    kw = dict(step_size=1800.0, window=3600, start_time=net["t0"], seed=8, **RULES[rule])
    sim = codes.Simulation(_graph(codes, net), M=replicas, iterations=14, path="batched", **kw)
    want = oracle.run(net["start"], net["end"], net["u"], net["v"], 71, n_replicas=replicas, n_steps=14, transition=0,
                      **kw)
    np.testing.assert_array_equal(sim.run(), want)


@pytest.mark.parametrize("replicas", [70, 1030])
def test_networks(codes, oracle, replicas):
    nets = [synthetic.tiny(seed=80 + k, n_nodes=n, n_contacts=8 * n) for k, n in enumerate((30, 180, 7, 65))]
    s, e, u, v, n, off = codes.batch_networks(nets)
    kw = dict(M=replicas, iterations=24, step_size=1800.0, window=1800, start_time=nets[0]["t0"], seed=13,
              transition="countdown", initial_count=3, infect_prob=0.3, exposed_duration=3600, infectious_duration=7200,
              resistant_duration=5400)
    got = codes.Simulation(codes.Graph.from_arrays(s, e, u, v, n), networks=off, path="batched", **kw).run()
    want = oracle.run(s, e, u, v, n, net_first=off, ncls_cap=0, **_oracle_kw(kw))
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("case", [0, 3])  # one and two bytes
def test_node_states(codes, oracle, case):
    net = synthetic.tiny(seed=31, n_nodes=30, n_contacts=300)
    kw = dict(COUNTDOWN_CASES[case], start_time=net["t0"], seed=3, transition="countdown")
    sim = codes.Simulation(_graph(codes, net), record_node_states=True, path="batched", **kw)
    seen = []
    counts = sim.run(node_states=lambda k, ts, st: seen.append(st) and 0)
    want_c, want_s = oracle.run(net["start"], net["end"], net["u"], net["v"], net["n_nodes"], node_states=True,
                                **_oracle_kw(kw))
    np.testing.assert_array_equal(counts, want_c)
    np.testing.assert_array_equal(np.stack(seen), want_s)


def test_the_table_takes_the_place_of_the_sets(codes):
    """One kernel a step (k_cd_step), where the plain path takes two."""
    net = synthetic.tiny(seed=1, n_nodes=1000, n_contacts=3000)
    sim = codes.Simulation(_graph(codes, net), M=320, iterations=100, path="batched", step_size=300.0, window=300,
                           start_time=net["t0"], initial_infected=0.1, infect_prob=0.2, exposed_duration=10_000,
                           infectious_duration=15_000, resistant_duration=0)
    plain = codes.Simulation(_graph(codes, net), M=320, iterations=100, path="plain", step_size=300.0, window=300,
                             start_time=net["t0"], initial_infected=0.1, infect_prob=0.2, exposed_duration=10_000,
                             infectious_duration=15_000, resistant_duration=0)
    np.testing.assert_array_equal(sim.run(), plain.run())
    assert sim.info["kernels_per_run"] < plain.info["kernels_per_run"]
