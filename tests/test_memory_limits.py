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
