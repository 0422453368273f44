"""The passes over all edges: the reverse CSR of the device graph, the 32-bit
parent recovery and the tree-edge lookup of the path costs, at the sizes
where they take another route: chunks of a warp and of the whole grid, long
runs of empty rows, a hub, one to nine distance-only objectives, distances
below and above 2^31. Whole numbers, compared with numpy and the oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
from gpu_util import assert_matches_oracle, dev, run_update_device  # noqa: E402


def graph(n, m, K, seed, hub=False, gaps=False, wmax=100):
    rng = np.random.default_rng(seed)
    tails = rng.integers(0, n, m)
    if gaps:  # edges leave only a few rows, far apart
        tails = tails // 997 * 997
    src, dst = np.concatenate([tails, np.arange(n - 1)]), np.concatenate([rng.integers(0, n, m), np.arange(1, n)])
    if gaps:
        src, dst = src[:m], dst[:m]
    if hub:
        src, dst = np.concatenate([src, np.zeros(n, int), np.arange(n)]), np.concatenate([dst, np.arange(n),
                                                                                         np.zeros(n, int)])
    ok = src != dst
    keys = np.unique(src[ok].astype(np.int64) * n + dst[ok])
    row = np.searchsorted(keys, np.arange(n + 1) * np.int64(n)).astype(np.int32)
    return row, (keys % n).astype(np.int32), rng.integers(1, wmax + 1, (len(keys), K)).astype(np.int32)


@pytest.mark.parametrize("n,m,K,hub,gaps", [(1, 0, 1, False, False), (2, 1, 1, False, False),
                                            (33, 31, 2, False, False), (1000, 5000, 3, False, False),
                                            (200000, 3000, 2, False, True), (5000, 20000, 4, True, False),
                                            (300000, 1300000, 3, True, False)])
def test_reverse_csr(n, m, K, hub, gaps):
    row, col, w = graph(n, m, K, n + m, hub, gaps)
    m = len(col)
    ws = mb.Workspace(timeout_ms=20000)
    out_w, in_w = dev(np.zeros(max(m * K, 1), np.int32)), dev(np.zeros(max(m * K, 1), np.int32))
    in_row, in_col = dev(np.zeros(n + 1, np.int32)), dev(np.zeros(max(m, 1), np.int32))
    for _ in range(2):  # the second build reuses the counters
        ws.build_device_graph(n, m, K, dev(row), dev(col), dev(w.reshape(-1)), out_w, in_row, in_col, in_w)
    ws.close()
    tail = np.repeat(np.arange(n), np.diff(row))
    assert np.array_equal(in_row.cpu().numpy(), np.concatenate([[0], np.cumsum(np.bincount(col, minlength=n))]))
    assert np.array_equal(out_w.cpu().numpy()[:m * K].reshape(K, m), w.T)
    # the order within a vertex's in-edges is not specified
    head = np.repeat(np.arange(n), np.diff(in_row.cpu().numpy()))
    got = np.column_stack([head, in_col.cpu().numpy()[:m], in_w.cpu().numpy()[:m * K].reshape(K, m).T])
    exp = np.column_stack([col, tail, w])
    assert np.array_equal(got[np.lexsort(got.T[::-1])], exp[np.lexsort(exp.T[::-1])])


@pytest.mark.parametrize("n,m,K,hub,gaps", [(100001, 1400003, 8, True, False), (900001, 1500000, 8, False, True),
                                            (100001, 2700000, 4, False, False), (50000, 8000000, 2, False, False)])
def test_reverse_csr_larger_than_l2_keeps(n, m, K, hub, gaps):
    """Reverse arrays of more than 48 MB, which are stored in order."""
    assert 4 * m * (K + 1) > 48 << 20
    test_reverse_csr(n, m, K, hub, gaps)


@pytest.mark.parametrize("high", [False, True])
@pytest.mark.parametrize("K", [1, 4, 5, 8, 9])
def test_full_recovery(K, high):
    """high: weights near 2^31, so that distances need more than 31 bits."""
    wmax = 2 ** 31 - 1 if high else 40
    g = mb.HostGraph.from_arrays(*graph(3000, 9000, K, 10 * K + high, hub=True, wmax=wmax))
    b = mb.HostBatch.generate(g, 400, seed=K, wmax=wmax)
    ws = mb.Workspace(timeout_ms=20000)
    # a bound that leaves no room for the parent next to the distance
    res = run_update_device(ws, g, b, max_weight=2 ** 60 // 3000)
    ws.close()
    assert all(st.packed_parents == 0 for st in res["stats"])
    assert_matches_oracle(res, g, b)
