"""Simulation.info's device_bytes against the device's free memory."""
import numpy as np
import pytest

from replay_b200 import synthetic

pytestmark = pytest.mark.gpu


# windows that list their rows in groups of 256 MB, windows by row pointers in two workspaces, windows kept
@pytest.mark.parametrize("contacts,csr", [(400_000, "per-step"), (6_000_000, "per-step"), (400_000, "prebuilt")])
def test_device_bytes_hold_every_buffer(contacts, csr):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    n, T = 1_500_000, 20
    rng = np.random.default_rng(4)
    u = rng.integers(0, n - 1, contacts).astype(np.int32)
    s = synthetic.EPOCH_2000 + rng.integers(0, T * 3600, contacts)
    g = rb.Graph.from_arrays(s, s + 600, u, u + 1, n)
    kw = dict(M=64, iterations=T, step_size=3600.0, window=3600, start_time=synthetic.EPOCH_2000, ncls_cap=False,
              transition="geometric", beta=1e-4, p_ei=0.1, p_ir=0.1, initial_count=3, csr=csr)
    rb.Simulation(g, **kw).close()  # the kernels are loaded
    rb.release_cached_memory()
    free = torch.cuda.mem_get_info()[0]
    sim = rb.Simulation(g, **kw)
    held = free - torch.cuda.mem_get_info()[0]
    # whole 2 MB pages for some 30 buffers, and the captured graph; scratch of the creation is kept apart
    rb.release_cached_memory()
    held = min(held, free - torch.cuda.mem_get_info()[0])
    assert held - (96 << 20) <= sim.info["device_bytes"] <= held
