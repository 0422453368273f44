"""Row records by the share of rows that are longer than one (4 edges): one in
50 or fewer use them. Both sides of the line, in updates, trees from scratch
and combined graphs, equal the oracle's."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
import oracle as orc  # noqa: E402
from gpu_util import assert_matches_oracle, run_update_device  # noqa: E402


@pytest.mark.parametrize("longer", [0, 1, 60, 61, 600])
def test_share_of_long_rows(longer):
    """3,000 vertices (the line: 60 longer rows) of two edges, `longer` of them
    of five to nine."""
    n, K = 3000, 3
    rng = np.random.default_rng(longer)
    degree = np.full(n, 2)
    degree[rng.choice(n, longer, replace=False)] = 5 + np.arange(longer) % 5
    row = np.concatenate([[0], np.cumsum(degree)]).astype(np.int32)
    col = np.concatenate([np.sort((v + np.concatenate([[1], 2 + rng.choice(60, d - 1, replace=False)])) % n)
                          for v, d in enumerate(degree)]).astype(np.int32)
    w = rng.integers(1, 60, (len(col), K)).astype(np.int32)
    g = mb.HostGraph.from_arrays(row, col, w)
    ws = mb.Workspace(timeout_ms=20000)
    dg = mb.DeviceGraph.upload(ws, g)
    d = torch.empty(n, dtype=torch.int64, device="cuda")
    p = torch.empty(n, dtype=torch.int32, device="cuda")
    for delta in (20, 10 ** 9):
        st = ws.sosp_from_scratch(n, g.m, dg.out_row, dg.out_col, dg.out_w[:g.m], 0, delta, 59, d, p)
        de, pe = orc.dijkstra(row, col, w, 0, 0)
        assert st.iterations == st.epochs  # (the asynchronous loop)
        assert np.array_equal(d.cpu().numpy(), de) and np.array_equal(p.cpu().numpy(), pe)
    for seed in range(3):
        # (deletions and insertions move rows across a record's length)
        b = mb.HostBatch.generate(g, 150, seed=seed, wmax=60)
        assert_matches_oracle(run_update_device(ws, g, b), g, b)
    ws.close()
