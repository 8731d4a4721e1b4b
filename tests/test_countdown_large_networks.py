"""The countdown rule on a network of more than 2^20 nodes that all change
class in the same steps: a step's change of a count does not fit the signed
half of its field."""
import ctypes as C

import numpy as np
import pytest

from replay_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes", [(1 << 20) + 1, (1 << 21) - 1])
@pytest.mark.parametrize("set_bytes", [1 << 34, 0])  # sets of replicas, codes
def test_all_nodes_change_together(nodes, set_bytes, monkeypatch):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    L = rb.lib()
    create = L.rp_sim_create_bounded
    create.argtypes, create.restype = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int32, C.c_int64, C.c_void_p], C.c_int
    monkeypatch.setattr(L, "rp_sim_create", lambda g, p, out: create(g, p, None, 1, set_bytes, out))
    s = np.array([synthetic.EPOCH_2000])
    g = rb.Graph.from_arrays(s, s + 60, [0], [1], nodes)
    kw = dict(M=3, iterations=9, step_size=600.0, window=600, start_time=synthetic.EPOCH_2000, initial_infected=1.0,
              infect_prob=0.0, exposed_duration=600, infectious_duration=1800, resistant_duration=1800)
    got = rb.Simulation(g, path="batched", **kw).run()
    monkeypatch.undo()
    np.testing.assert_array_equal(got, rb.Simulation(g, path="plain", **kw).run())
    assert (got.sum(axis=2) == nodes).all() and got.max() == nodes
