"""Rows around the thresholds of the bulk loop's whole-CTA rows (more than 512
edges, in a graph with a row of more than 2,048), and more such rows than the
queue of a CTA holds: 300 of them under one hub, with the whole grid and with
two CTAs, whose pull and first iteration meet all 300 at once. Whole numbers:
every result equals the oracle's."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
import oracle as orc  # noqa: E402
from gpu_util import assert_matches_oracle, run_update_device  # noqa: E402


def hubs(top, deg, K, rng):
    """Vertex 0 with `top` edges, the first 300 of them to vertices with
    `deg` edges each (a ring over the other vertices, both directions)."""
    n = 301 + max(top, 1200)
    src, dst = [np.zeros(top, np.int64)], [np.arange(1, top + 1)]
    for h in range(1, 301):
        far = 301 + (np.arange(deg) + 7 * h) % (n - 301)
        src += [np.full(deg, h), far]
        dst += [far, np.full(deg, h)]
    key = np.unique(np.concatenate(src) * n + np.concatenate(dst))
    row = np.searchsorted(key, np.arange(n + 1) * n).astype(np.int32)
    return row, (key % n).astype(np.int32), rng.integers(1, 200, (len(key), K)).astype(np.int32)


@pytest.mark.parametrize("ctas", [0, 2])
@pytest.mark.parametrize("top,deg", [(2048, 513), (2049, 511), (2049, 512), (2049, 513), (5000, 1100)])
def test_rows_around_the_thresholds(top, deg, ctas):
    rng = np.random.default_rng(top + deg)
    row, col, w = hubs(top, deg, 2, rng)
    assert (np.diff(row)[1:301] == deg).all() and row[1] == top
    g = mb.HostGraph.from_arrays(row, col, w)
    ws = mb.Workspace(timeout_ms=20000)
    ws.set_grid(ctas)
    for mode, seed in (("targeted", 3), ("uniform", 4)):
        b = mb.HostBatch.generate(g, 3000, 40.0, mode, 0, False, seed, 0, 1, 200)
        assert_matches_oracle(run_update_device(ws, g, b, pref=[1, 2]), g, b, pref=[1, 2])
    w0 = np.ascontiguousarray(w[:, :1])
    g = mb.HostGraph.from_arrays(row, col, w0)
    dg = mb.DeviceGraph.upload(ws, g)
    d = torch.empty(g.n, dtype=torch.int64, device="cuda")
    p = torch.empty(g.n, dtype=torch.int32, device="cuda")
    ws.sosp_from_scratch(g.n, g.m, dg.out_row, dg.out_col, dg.out_w, 0, 60, 200, d, p)
    de, pe = orc.dijkstra(row, col, w0, 0, 0)
    assert np.array_equal(d.cpu().numpy(), de) and np.array_equal(p.cpu().numpy(), pe)
    ws.close()
