"""Closing a handle with a block above the kept blocks' total (8 GiB) frees
that block and keeps the others."""
import numpy as np
import pytest

from replay_b200 import synthetic

pytestmark = pytest.mark.gpu


def test_a_block_above_the_limit_leaves_the_others_kept():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    if torch.cuda.mem_get_info()[0] < 24 << 30:
        pytest.skip("needs 24 GB free")
    n, T = 20_000, 1000
    s = np.array([synthetic.EPOCH_2000, synthetic.EPOCH_2000 + 40])
    g = rb.Graph.from_arrays(s, s + 300, [0, 1], [1, 2], n)
    kw = dict(M=4096, step_size=60.0, window=60, start_time=synthetic.EPOCH_2000, path="batched", infect_prob=0.1,
              initial_infected=0.1, exposed_duration=600, infectious_duration=600, resistant_duration=100_000_000)
    rb.release_cached_memory()
    free0 = torch.cuda.mem_get_info()[0]
    rb.Simulation(g, iterations=40, **kw).close()
    kept = free0 - torch.cuda.mem_get_info()[0]
    assert kept > 200 << 20  # 41 sets of 10 MB
    # 900 steps until the resistance ends: sets of 9.4 GB in one block
    kw.update(exposed_duration=24_000, infectious_duration=30_000, resistant_duration=0)
    sim = rb.Simulation(g, iterations=T, **kw)
    assert sim.info["device_bytes"] > 8 << 30
    sim.close()
    assert free0 - torch.cuda.mem_get_info()[0] >= kept - (32 << 20)
    g.close()
    rb.release_cached_memory()
