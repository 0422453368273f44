"""The bulk loop's queue of rows for the whole CTA, with more rows than it
holds in one iteration: hundreds of rows above the CTA threshold and a few
hubs, expanded by one CTA. Equal to the asynchronous loop, and the hubs are not
left to a warp each (which takes milliseconds)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
from gpu_util import dev  # noqa: E402


@pytest.mark.parametrize("mids,edges", [(60, 600), (300, 600), (450, 2000), (300, 512), (300, 513)])
def test_hubs_among_many_long_rows(mids, edges):
    rng = np.random.default_rng(mids + edges)
    hubs, hub_edges, leaves = 6, 150000, mids * 100
    first = 1 + mids + hubs
    n = first + leaves
    degrees = np.concatenate([[mids + hubs], np.full(mids, edges), np.full(hubs, hub_edges), np.zeros(leaves, int)])
    row = np.concatenate([[0], np.cumsum(degrees)]).astype(np.int32)
    order = rng.permutation(np.arange(1, first))  # rows and hubs in any order
    col = np.concatenate([order, rng.integers(first, n, degrees[1:].sum())]).astype(np.int32)
    w = rng.integers(1, 100, len(col)).astype(np.int32)
    w[:mids + hubs] = 1
    ws = mb.Workspace(timeout_ms=20000)
    graph = [dev(x) for x in (row, col, w)]
    out, best = [], []
    for hub_row in (0, 2048, 1 << 30):
        ws.set_grid(0, hub_row)  # 2048: only the hubs go to the CTA; 2^30: no hub rows, the asynchronous loop
        dist, par = torch.zeros(n, dtype=torch.int64, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
        times = []
        for _ in range(6):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            ws.sosp_from_scratch(n, len(col), *graph, 0, 1000, 100, dist, par)
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end))
        out.append((dist, par))
        best.append(min(times[2:]))
    ws.close()
    for d, p in out[1:]:
        assert torch.equal(d, out[0][0]) and torch.equal(p, out[0][1])
    assert best[0] < 1.5 * best[1], best
