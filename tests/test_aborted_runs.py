"""A run that its callback ends early leaves nothing behind: the next run of
the same simulation gives every count.  The windows are built in several
groups, so that the next group's build is under way when the callback ends the
run."""
import numpy as np
import pytest

from replay_b200 import synthetic

pytestmark = pytest.mark.gpu

RULES = [dict(transition="geometric", beta=1e-3, p_ei=0.2, p_ir=0.1, initial_infected=0.05),
         dict(transition="countdown", infect_prob=0.4, exposed_duration=3600, infectious_duration=14400,
              resistant_duration=3600, initial_infected=0.05)]


@pytest.mark.parametrize("rule", range(len(RULES)))
@pytest.mark.parametrize("contacts", [400_000, 40_000])  # a window's rows by row pointers, and listed
def test_next_run_after_an_abort(rule, contacts):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    n, T = 150_000, 16
    rng = np.random.default_rng(rule)
    u = rng.integers(0, n // 8, contacts).astype(np.int32)
    v = ((u + rng.integers(1, n, contacts)) % n).astype(np.int32)
    s = synthetic.EPOCH_2000 + rng.integers(0, T * 3600, contacts)
    g = rb.Graph.from_arrays(s, s + rng.integers(1, 3600, contacts), u, v, n)
    kw = dict(M=32, iterations=T, step_size=3600.0, window=3600, start_time=synthetic.EPOCH_2000, seed=3, ncls_cap=False,
              path="batched", **RULES[rule])
    want = rb.Simulation(g, **kw).run()
    sim = rb.Simulation(g, record_node_states=True, **kw)
    for stop in (0, 1, 2, 5, 12):
        with pytest.raises(rb.ReplayError, match="aborted"):
            sim.run(lambda k, ts, states: k == stop)
        np.testing.assert_array_equal(sim.run(lambda k, ts, states: False), want)
        with pytest.raises(rb.ReplayError, match="aborted"):
            sim.run_text(lambda k, ts, data: k == stop)
        sim.enqueue()
        np.testing.assert_array_equal(sim.counts(), want)
