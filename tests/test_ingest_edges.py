"""The device passes of the index build where they can go wrong: contact
counts around the 16-contact threads and 4,096-contact chunks of the nesting
count, long nesting chains and ties across chunks, endpoints in any order and
out of range, and window plans over every duration class."""
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


@pytest.mark.parametrize("n", [1, 15, 16, 17, 4095, 4096, 4097, 12289])
@pytest.mark.parametrize("shape", ["mixed", "chain", "ties"])
def test_sublist_count(oracle, n, shape):
    rb = _rb()
    rng = np.random.default_rng(n)
    t0 = synthetic.EPOCH_2000
    if shape == "mixed":
        start = t0 + rng.integers(0, 50_000, n)
        end = start + rng.integers(1, 9_000, n)
    elif shape == "chain":  # each inside the one before, then a second chain
        k = np.arange(n)
        start = t0 + np.where(k < n // 2, k, 200_000 + k)
        end = t0 + np.where(k < n // 2, 100_000 - k, 500_000 - k)
    else:
        start = t0 + rng.integers(0, 5, n)
        end = start + rng.integers(1, 4, n)
    u = rng.integers(0, 40, n).astype(np.int32)
    v = ((u + 1 + rng.integers(0, 39, n)) % 40).astype(np.int32)  # u > v as often as not
    g = rb.Graph.from_arrays(start, end, u, v, 47)
    info = g.info
    assert info["nlists"] == oracle.sorted_index(start, end, np.minimum(u, v), np.maximum(u, v))[5]
    assert info["n_index"] == len(np.unique(np.concatenate([u, v])))


@pytest.mark.parametrize("at,u,v", [(0, -1, 2), (5, 3, 7), (4999, 2, 2_000_000_000)])
def test_first_contact_out_of_range_is_named(at, u, v):
    rb = _rb()
    n = 5000
    uu, vv = np.zeros(n, np.int32), np.ones(n, np.int32)
    uu[at], vv[at] = u, v
    uu[at + 1:at + 3] = 7  # later ones are not the first
    with pytest.raises(rb.ReplayError, match=f"contact {at} joins"):
        rb.Graph.from_arrays(np.arange(n), np.arange(n) + 5, uu, vv, 7)


@pytest.mark.parametrize("sign", [1, -1])
def test_plans_cover_every_duration_class(oracle, sign):
    rb = _rb()
    rng = np.random.default_rng(2)
    dur = np.concatenate([[0, -3], 2 ** np.arange(0, 30), 2 ** np.arange(1, 30) + 1, 2 ** np.arange(2, 30) - 1])
    start = sign * 1_000_000 + rng.integers(0, 4000, len(dur))
    end = start + dur
    u = rng.integers(0, 9, len(dur)).astype(np.int32)
    v = u + 1
    g = rb.Graph.from_arrays(start, end, u, v, 10)
    ss, se, su, sv, perm, nl = oracle.sorted_index(start, end, u, v)
    for ws in (sign * 1_000_000 - 5000, sign * 1_000_000, sign * 1_000_000 + 1000, sign * 1_000_000 + 100_000):
        for cap in (True, False):
            rp, col, val, nh = rb.window_csr(g, ws, ws + 777, 1.0, "f32", cap)
            hits = oracle.window_hits(ss, se, nl if cap else len(ss), ws, ws + 777)
            orp, ocol, oval = oracle.csr_f32(ss, se, su, sv, hits, 10, ws, ws + 777, np.float32(1))
            assert nh == len(hits)
            np.testing.assert_array_equal(rp, orp)
            np.testing.assert_array_equal(col, ocol)
            np.testing.assert_array_equal(val.view(np.int32), oval.view(np.int32))
