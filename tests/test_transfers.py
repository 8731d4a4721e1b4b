"""Large host copies through staging buffers: contact arrays and counts around
the chunk size, several threads at once, pinned arrays, and after the cached
memory was given back."""
import threading

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


def _net(n, seed):
    rng = np.random.default_rng(seed)
    u = rng.integers(0, 500, n).astype(np.int32)
    v = ((u + 1 + rng.integers(0, 499, n)) % 501).astype(np.int32)
    s = synthetic.EPOCH_2000 + rng.integers(0, 86400, n)
    return s, s + rng.integers(1, 3000, n), u, v


def _total(rb, net, ws):
    """Contact-seconds of a window from the CSR and from the arrays."""
    s, e, u, v = net
    g = rb.Graph.from_arrays(s, e, u, v, 501)
    val = rb.window_csr(g, ws, ws + 3600, weight="i32", ncls_cap=False)[2]
    g.close()
    over = np.clip(np.minimum(e, ws + 3600) - np.maximum(s, ws), 0, None).sum()
    return int(val.astype(np.int64).sum()), 2 * int(over)


# 4 MB of int64 is the smallest staged array; 2 MB chunks and a remainder
@pytest.mark.parametrize("n", [524_287, 524_288, 786_433, 3_000_001])
def test_uploads(n):
    rb = _rb()
    for k in range(2):
        got, want = _total(rb, _net(n, n + k), synthetic.EPOCH_2000 + 7200)
        assert got == want
        rb.release_cached_memory()


def test_uploads_of_several_threads_and_pinned_arrays():
    import torch
    rb = _rb()
    out = {}

    def one(k):
        out[k] = _total(rb, _net(900_000, k), synthetic.EPOCH_2000 + 3600 * (k + 1))

    ts = [threading.Thread(target=one, args=(k,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert len(out) == 4 and all(a == b for a, b in out.values())
    net = [torch.from_numpy(a).pin_memory().numpy() for a in _net(900_000, 9)]
    got, want = _total(rb, net, synthetic.EPOCH_2000)
    assert got == want


# rows x replicas x 16 bytes: below and above 4 MB, with a remainder of a chunk
@pytest.mark.parametrize("steps,replicas", [(40, 6000), (60, 6000), (99, 9999)])
def test_downloads(oracle, steps, replicas):
    rb = _rb()
    net = synthetic.tiny(seed=160, n_nodes=30, n_contacts=300, span=steps * 600)
    g = rb.Graph.from_arrays(net["start"], net["end"], net["u"], net["v"], 30)
    kw = dict(step_size=600.0, window=600, start_time=net["t0"], seed=2, beta=1e-3, p_ei=0.1, p_ir=0.05, initial_count=2)
    sim = rb.Simulation(g, M=replicas, iterations=steps, transition="geometric", **kw)
    counts = sim.run()
    assert (counts.sum(axis=2) == 30).all()
    np.testing.assert_array_equal(sim.counts(), counts)
    # the last replicas alone, against the oracle
    off = replicas // 32 * 32 - 32
    want = oracle.run(net["start"], net["end"], net["u"], net["v"], 30, n_replicas=32, n_steps=steps, transition=1,
                      replica_offset=off, **kw)
    np.testing.assert_array_equal(counts[:, off:off + 32], want)
