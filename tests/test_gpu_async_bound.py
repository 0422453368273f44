"""Distances next to what a packed word holds: the asynchronous loop adds a
weight to a word without a check, so a launch whose bound is within 2^31 of the
word runs the bulk loop. The graph's distances reach the bound, and the edges
that leave its far end would wrap a word around to a small distance."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
import oracle as orc  # noqa: E402


@pytest.mark.parametrize("weight,asynchronous", [(2 ** 30 - 100, True), (2 ** 30 + 16000, False)])
def test_distances_at_the_bound(weight, asynchronous):
    """A chain of 131,071 vertices (17 parent bits, distances below 2^47) of
    equal weights, and an edge of that weight from each of the last 64 vertices
    back to the first ones."""
    n = 2 ** 17 - 1
    assert mb.choose_packing(n, weight)[0] == 17
    most = weight * (n - 1)
    assert (most + 2 ** 31 <= 2 ** 47 - 1) == asynchronous
    assert (most + weight >= 2 ** 47) != asynchronous  # the far end's edges wrap
    tail = np.concatenate([np.arange(n - 1), np.arange(n - 64, n)])
    head = np.concatenate([np.arange(1, n), np.arange(1, 65)])
    order = np.lexsort((head, tail))
    row = np.searchsorted(tail[order], np.arange(n + 1)).astype(np.int32)
    col = head[order].astype(np.int32)
    w = np.full((len(col), 1), weight, np.int32)
    g = mb.HostGraph.from_arrays(row, col, w)
    ws = mb.Workspace(timeout_ms=20000)
    dg = mb.DeviceGraph.upload(ws, g)
    d = torch.empty(n, dtype=torch.int64, device="cuda")
    p = torch.empty(n, dtype=torch.int32, device="cuda")
    st = ws.sosp_from_scratch(n, g.m, dg.out_row, dg.out_col, dg.out_w[:g.m], 0, 10 ** 12, weight, d, p)
    de, pe = orc.dijkstra(row, col, w, 0, 0)
    assert int(de.max()) == most
    assert np.array_equal(d.cpu().numpy(), de) and np.array_equal(p.cpu().numpy(), pe)
    # (the bulk loop counts its iterations and its thresholds apart)
    assert (st.iterations == st.epochs) == asynchronous
    ws.close()
