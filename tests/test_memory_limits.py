"""Calls on a device whose memory is nearly taken."""
import contextlib

import numpy as np
import pytest

from replay_b200 import synthetic

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _rb():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200
    return replay_b200


@contextlib.contextmanager
def memory_left(rb, nbytes):
    """About nbytes of device memory free (whole 2 MB pages) and no kept blocks."""
    import torch
    rb.release_cached_memory()
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    held = torch.empty(max(0, torch.cuda.mem_get_info()[0] - int(nbytes)) // (2 * MB) * (2 * MB), dtype=torch.uint8,
                       device="cuda")
    try:
        yield
    finally:
        del held
        rb.release_cached_memory()
        torch.cuda.empty_cache()


def test_argument_error_before_the_memory_error():
    """A contact with an endpoint out of range is an argument error (1) whether or not the index would fit (4)."""
    rb = _rb()
    n = 10_000_000
    s = np.full(n, synthetic.EPOCH_2000)
    u, v = np.zeros(n, np.int32), np.ones(n, np.int32)
    rb.Graph.from_arrays(s[:9], s[:9] + 5, u[:9], v[:9], 2).close()
    with memory_left(rb, 128 * MB):  # the contacts take 280 MB
        with pytest.raises(rb.ReplayError) as e:
            rb.Graph.from_arrays(s, s + 5, u, v, 2)
        assert e.value.status == 4
        v[n - 3] = 2
        with pytest.raises(rb.ReplayError, match=f"contact {n - 3} joins") as e:
            rb.Graph.from_arrays(s, s + 5, u, v, 2)
        assert e.value.status == 1


def test_sets_of_replicas_leave_room_or_give_way():
    """Countdown sets of 1.6 GB in ever less memory: every replay whose codes (200 MB) fit is accepted and
    gives the same counts."""
    rb = _rb()
    n, T, M = 20_000, 160, 4096
    rng = np.random.default_rng(2)
    u = rng.integers(0, n - 1, 200_000).astype(np.int32)
    s = synthetic.EPOCH_2000 + rng.integers(0, T * 600, len(u))
    g = rb.Graph.from_arrays(s, s + 400, u, u + 1, n)
    kw = dict(M=M, iterations=T, step_size=600.0, window=600, start_time=synthetic.EPOCH_2000, path="batched", seed=2,
              initial_infected=0.02, infect_prob=0.5, exposed_duration=30_000, infectious_duration=60_000,
              resistant_duration=0)
    sim = rb.Simulation(g, **kw)
    want = sim.run()
    full = sim.info["device_bytes"]
    assert full > 1600 * MB
    sim.close()
    # from all the sets would take and more, over every size at which a part of them does not fit, to the codes alone
    tight = full - 1600 * MB + 200 * MB + 192 * MB
    taken = []
    for left in [full + 900 * MB, full + 400 * MB, *range(full + 64 * MB, full - 64 * MB, -8 * MB), 1200 * MB, tight]:
        with memory_left(rb, left):
            sim = rb.Simulation(g, **kw)
            taken.append(sim.info["device_bytes"] == full)
            if left in (full + 64 * MB, tight):
                np.testing.assert_array_equal(sim.run(), want)
            sim.close()
    assert taken[0] and not any(taken[1:])


def test_kept_states_leave_room_or_give_way():
    """Mean-field states of 2.4 GB in ever less memory: every replay whose checkpoints (0.4 GB) fit is accepted and
    gives the same values and gradients, bit for bit for the nodes."""
    rb = _rb()
    import torch
    from replay_b200.meanfield import MeanField
    n, T = 500_000, 200
    rng = np.random.default_rng(2)
    u = rng.integers(0, n - 1, 400_000).astype(np.int32)
    s = synthetic.EPOCH_2000 + rng.integers(0, T * 600, len(u))
    g = rb.Graph.from_arrays(s, s + 400, u, u + 1, n)
    x0 = torch.zeros(4, n, device="cuda")
    x0[0], x0[2] = 0.9, 0.1
    x0.requires_grad_()

    def passes(left):
        """Forward and gradient with `left` bytes free before the creation; the bytes that it took."""
        with memory_left(rb, left):
            free = torch.cuda.mem_get_info()[0]
            mf = MeanField(g, iterations=T, step_size=600.0, window=600, start_time=synthetic.EPOCH_2000)
            took = free - torch.cuda.mem_get_info()[0]
            inc, xT = mf(x0, 3e-4, p_ei=0.03, p_ir=0.02)
            (grad,) = torch.autograd.grad(xT[3].sum(), x0)
            mf.close()
            return took, xT.detach().cpu().numpy(), grad.cpu().numpy()

    full, want, want_grad = passes(16 << 30)
    assert full > 2600 * MB  # states and the windows' row pointers
    kept = []
    sizes = [full + 900 * MB, full + 400 * MB, *range(full + 128 * MB, full - 64 * MB, -16 * MB), full - 1400 * MB]
    for left in sizes:
        took, xT, grad = passes(left)
        kept.append(took > full - 1000 * MB)
        np.testing.assert_array_equal(xT, want)
        np.testing.assert_array_equal(grad, want_grad)
    assert kept[0] and not any(kept[1:])


# windows in groups of 256 MB that list their rows; a window's contacts, mostly the same pairs over and over, in an
# arena with room for every contact
@pytest.mark.parametrize("csr,nodes,pairs,contacts,T", [("per-step", 1_500_000, 1_499_999, 400_000, 20),
                                                        ("prebuilt", 2_000, 50, 6_000_000, 100)])
def test_windows_give_room_up(csr, nodes, pairs, contacts, T):
    """In ever less memory, down to what one window at a time takes, a replay is accepted and gives the same counts."""
    rb = _rb()
    rng = np.random.default_rng(5)
    u = rng.integers(0, pairs, contacts).astype(np.int32)
    s = synthetic.EPOCH_2000 + rng.integers(0, T * 3600, contacts)
    g = rb.Graph.from_arrays(s, s + 300, u, u + 1, nodes)
    kw = dict(M=64, iterations=T, step_size=3600.0, window=3600, start_time=synthetic.EPOCH_2000, ncls_cap=False,
              transition="geometric", beta=1e-4, p_ei=0.1, p_ir=0.1, initial_count=nodes // 20, seed=1, csr=csr)
    sim = rb.Simulation(g, **kw)
    want, full = sim.run(), sim.info["device_bytes"]
    sim.close()
    least = 200 * MB if csr == "per-step" else full - 48 * MB
    held = []
    for left in np.linspace(full + 192 * MB, least, 24):
        with memory_left(rb, left):
            sim = rb.Simulation(g, **kw)
            held.append(sim.info["device_bytes"])
            np.testing.assert_array_equal(sim.run(), want)
            sim.close()
    assert held[0] == full and held[-1] < full - 48 * MB


def text(sim):
    lines = []
    sim.run_text(lambda k, ts, data: lines.append((k, data)) and None)
    return lines


def test_text_takes_the_place_of_small_sets():
    """Sets up to 256 MB are taken without a look at what stays free: the first text run turns them into codes."""
    rb = _rb()
    n = 20_000
    s = np.array([synthetic.EPOCH_2000])
    g = rb.Graph.from_arrays(s, s + 900, [0], [1], n)
    kw = dict(M=512, iterations=150, step_size=600.0, window=600, start_time=synthetic.EPOCH_2000, path="batched",
              initial_infected=0.1, infect_prob=0.1, exposed_duration=30_000, infectious_duration=50_000,
              resistant_duration=0, record_node_states=True)

    def first_lines(sim):
        lines = []

        def write(k, ts, data):
            lines.append(data)
            return k == 2
        with pytest.raises(rb.ReplayError, match="aborted"):
            sim.run_text(write)
        return lines
    sim = rb.Simulation(g, **kw)
    want, full = first_lines(sim), sim.info["device_bytes"]
    sim.close()
    sets = 132 * n * 64
    with memory_left(rb, full - sets + 110 * MB):  # the sets, and no room for the text's 128 MB
        sim = rb.Simulation(g, **kw)
        assert first_lines(sim) == want
        assert sim.info["device_bytes"] < full - sets // 2
        sim.close()


def test_text_after_a_call_without_memory():
    """run_text allocates its buffers at the first call; one that got only a part of them is refused, and so is the
    next, until there is memory."""
    rb = _rb()
    n, M = 20_000, 64
    s = np.array([synthetic.EPOCH_2000])
    g = rb.Graph.from_arrays(s, s + 900, [0], [1], n)
    kw = dict(M=M, iterations=2, step_size=1800.0, window=1800, start_time=synthetic.EPOCH_2000, transition="geometric",
              beta=1e-3, p_ir=0.1, initial_infected=0.1, record_node_states=True)
    want = text(rb.Simulation(g, **kw))
    assert sum(len(d) for _, d in want) > 3 * n * M * 20
    sim = rb.Simulation(g, **kw)
    with memory_left(rb, 100 * MB):  # twice 64 MB of text
        for _ in range(2):
            with pytest.raises(rb.ReplayError) as e:
                text(sim)
            assert e.value.status == 4
    assert text(sim) == want
