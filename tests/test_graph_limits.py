"""Graphs at the limits of what their creation accepts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rb():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200
    return replay_b200


# the count of the nodes that appear strides over 2 GB of marks; from 2^31 - 606,208 nodes on the last stride
# passes the largest 32-bit index
@pytest.mark.parametrize("nodes", [2**31 - 1 - 148 * 16 * 256, 2**31 - 1])
def test_most_nodes(nodes):
    rb = _rb()
    last = nodes - 1
    g = rb.Graph.from_arrays([5, 9, 9], [8, 20, 30], np.array([0, last, last], np.int32),
                             np.array([last, 7, last - 1], np.int32), nodes)
    assert (g.info["n_nodes"], g.info["n_index"], g.info["n_contacts"]) == (nodes, 4, 3)
    g.close()
    rb.release_cached_memory()
