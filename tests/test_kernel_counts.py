"""kernels_per_run and profile()'s kernels count every launch of a replay."""
import pytest

from replay_b200 import synthetic

pytestmark = pytest.mark.gpu

GEOMETRIC = dict(transition="geometric", beta=1e-3, p_ei=0.2, p_ir=0.1)
COUNTDOWN = dict(transition="countdown", infect_prob=0.4, exposed_duration=1800, infectious_duration=3600,
                 resistant_duration=1800)
# init, bitmaps, counts and the final sums; init, the initial set's items and its change, and the final sums
BEFORE_AND_AFTER = 4


@pytest.mark.parametrize("rule", [GEOMETRIC, COUNTDOWN, dict(COUNTDOWN, resistant_duration=0, exposed_duration=0)])
@pytest.mark.parametrize("initial", [dict(initial_infected=0.1), dict(initial_count=4)])
def test_kernels_of_a_replay(rule, initial):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    net = synthetic.tiny(seed=160, n_nodes=50, n_contacts=2000, span=8 * 3600)
    g = rb.Graph.from_arrays(net["start"], net["end"], net["u"], net["v"], 50)
    kw = dict(M=70, path="batched", step_size=1800.0, window=1800, start_time=net["t0"], **rule, **initial)
    for T in (0, 1, 9):
        sim = rb.Simulation(g, iterations=T, **kw)
        said = sim.info["kernels_per_run"]
        if T == 0:
            assert said == BEFORE_AND_AFTER + (2 if "initial_count" in initial else 0)
        assert sim.profile()["kernels"] == said
