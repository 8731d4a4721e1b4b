"""Layouts with more replicas than the other files reach, against the oracle:
windows that list their rows with a second slice of columns (more than 4,096
replicas), and the countdown rule on several networks with rows of 32 words and
more (k_cd_flow's counters per network)."""
import numpy as np
import pytest

from replay_b200 import synthetic

pytestmark = pytest.mark.gpu


def _rb():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200
    return replay_b200


@pytest.mark.parametrize("replicas", [4097, 4130])
def test_listed_rows_with_a_second_slice(oracle, replicas):
    rb = _rb()
    n, T = 5000, 6
    rng = np.random.default_rng(3)
    # 60 contacts a window, a row of 60 pairs and one of 300 in some of them
    u = np.concatenate([rng.integers(0, n - 1, 60 * T), np.full(60, 5), np.full(300, 9)]).astype(np.int32)
    v = np.concatenate([u[:60 * T] + 1, 6 + rng.integers(0, 900, 60), 10 + rng.integers(0, 900, 300)]).astype(np.int32)
    s = synthetic.EPOCH_2000 + np.concatenate([rng.integers(0, T * 900, 60 * T), rng.integers(1800, 2000, 60),
                                               np.full(300, 3000)])
    e = s + rng.integers(1, 600, len(s))
    kw = dict(step_size=900.0, window=900, start_time=synthetic.EPOCH_2000, seed=4, beta=3e-3, p_ei=0.3, p_ir=0.05,
              initial_infected=0.1)
    g = rb.Graph.from_arrays(s, e, u, v, n)
    sim = rb.Simulation(g, M=replicas, iterations=T, path="batched", transition="geometric", ncls_cap=False, **kw)
    assert 8 * sim.info["max_candidates"] < n
    want = oracle.run(s, e, u, v, n, n_replicas=replicas, n_steps=T, transition=1, ncls_cap=0, **kw)
    assert (want[1:, :, 0] > 0).any()
    np.testing.assert_array_equal(sim.run(), want)


@pytest.mark.parametrize("replicas", [1000, 1030, 1100, 4130])
@pytest.mark.parametrize("csr", ["per-step", "prebuilt"])
def test_countdown_on_several_networks(oracle, replicas, csr):
    rb = _rb()
    nets = [synthetic.tiny(seed=80 + k, n_nodes=n, n_contacts=8 * n) for k, n in enumerate((30, 110, 7, 65))]
    s, e, u, v, n, off = rb.batch_networks(nets)
    kw = dict(step_size=1800.0, window=1800, start_time=nets[0]["t0"], seed=13, initial_count=3, infect_prob=0.4,
              exposed_duration=3600, infectious_duration=7200, resistant_duration=5400)
    sim = rb.Simulation(rb.Graph.from_arrays(s, e, u, v, n), networks=off, path="batched", csr=csr, M=replicas,
                        iterations=20, **kw)
    want = oracle.run(s, e, u, v, n, net_first=off, ncls_cap=0, n_replicas=replicas, n_steps=20, transition=0, **kw)
    np.testing.assert_array_equal(sim.run(), want)
    np.testing.assert_array_equal(sim.run(), want)
