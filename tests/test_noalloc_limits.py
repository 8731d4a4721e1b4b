"""rp_window_csr_noalloc plans its window in the stream: windows with and
without candidates, under a hit cap, at and above the most candidates it takes
(131,072), against rp_window_csr; a refused call writes nothing."""
import ctypes as C

import numpy as np
import pytest

from replay_b200 import synthetic

pytestmark = pytest.mark.gpu

T0 = synthetic.EPOCH_2000


def _call(L, g, ws, we, kind, cap, rp, ent):
    import torch
    nnz, nh = C.c_int64(-1), C.c_int64(-1)
    st = L.rp_window_csr_noalloc(g._h, ws, we, 0.5, kind, cap, rp.data_ptr(), ent.data_ptr(), len(ent) // 2,
                                 C.byref(nnz), C.byref(nh), torch.cuda.current_stream().cuda_stream)
    return st, nnz.value, nh.value


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("cap", [0, 1])
def test_windows(kind, cap):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    L = rb.lib()
    n, most = 3000, 131_072
    rng = np.random.default_rng(7)
    # hour 0: as many contacts as a window takes, hour 2: one more, hour 4: few of many durations, before hour 0: none
    u = rng.integers(0, n - 1, 2 * most + 1 + 900).astype(np.int32)
    v = (u + rng.integers(1, n, len(u))) % n
    s = np.concatenate([T0 + rng.integers(0, 3000, most), T0 + 7200 + rng.integers(0, 3000, most + 1),
                        T0 + 14400 + rng.integers(0, 3000, 900)])
    e = s + np.concatenate([rng.integers(1, 60, 2 * most + 1), 2 ** rng.integers(0, 12, 900)])
    g = rb.Graph.from_arrays(s, e, u, v, n)
    rp = torch.full((n + 1,), -7, dtype=torch.int32, device="cuda")
    ent = torch.full((4 * most,), -7, dtype=torch.int32, device="cuda")
    for ws, we in [(T0, T0 + 3600), (T0 + 14400, T0 + 18000), (T0 - 9000, T0 - 3600), (T0 + 15000, T0 + 15001)]:
        rp.fill_(-7), ent.fill_(-7)
        st, nnz, nh = _call(L, g, ws, we, kind, cap, rp, ent)
        assert st == 0, L.rp_last_error()
        want = rb.window_csr(g, ws, we, 0.5, "i32" if kind else "f32", bool(cap))
        assert nnz == len(want[1]) and nh == want[3]
        got = ent.cpu().numpy()
        np.testing.assert_array_equal(rp.cpu().numpy(), want[0])
        np.testing.assert_array_equal(got[:2 * nnz:2], want[1])
        np.testing.assert_array_equal(got[1:2 * nnz:2], want[2].view(np.int32))
        assert (got[2 * nnz:] == -7).all()
    rp.fill_(-7), ent.fill_(-7)
    st, nnz, nh = _call(L, g, T0 + 7200, T0 + 10800, kind, cap, rp, ent)
    assert st == 6 and b"131073 candidate" in L.rp_last_error()
    torch.cuda.synchronize()
    assert (nnz, nh) == (-1, -1) and (rp == -7).all() and (ent == -7).all()
    few = ent[:20].clone()  # too little room: the row pointers and the numbers, no pairs
    st, nnz, nh = _call(L, g, T0 + 14400, T0 + 18000, kind, cap, rp, few)
    assert st == 6 and nnz == int(rp[n]) > 10 and (few == -7).all()
