"""The pull pass's two orders of the candidates, on both sides of each of
their edges: fewer than a warp, one more than a tile of every CTA, and several
tiles; graphs with and without hub rows; the whole grid and one CTA. Trees
equal the oracle's."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
from gpu_util import assert_matches_oracle, run_update_device  # noqa: E402


@pytest.mark.parametrize("ctas", [0, 1, 5])
@pytest.mark.parametrize("hubs", [False, True])
@pytest.mark.parametrize("changes", [4, 1023, 1025, 5121, 20000])
def test_candidates_of_a_batch(changes, hubs, ctas):
    """Insertions only: the candidates are their heads, fewer than half of the
    vertices, so the pass pulls."""
    rng = np.random.default_rng(changes + hubs)
    n, K = 60000, 2
    tail = np.concatenate([rng.integers(0, n, 2 * n), np.arange(n - 1)])
    head = np.concatenate([rng.integers(0, n, 2 * n), np.arange(1, n)])
    if hubs:  # 3,000 edges into and out of two vertices
        tail = np.concatenate([tail, rng.integers(0, n, 3000), np.full(3000, 7)])
        head = np.concatenate([head, np.full(3000, 11), rng.integers(0, n, 3000)])
    keys = np.unique(tail[tail != head] * np.int64(n) + head[tail != head])
    row = np.searchsorted(keys, np.arange(n + 1) * np.int64(n)).astype(np.int32)
    col = (keys % n).astype(np.int32)
    g = mb.HostGraph.from_arrays(row, col, rng.integers(50, 100, (len(col), K)).astype(np.int32))
    to = rng.choice(n - 1, changes, replace=False) + 1
    b = mb.HostBatch.from_arrays(K, (to + rng.integers(1, n, changes)) % n, to,
                                 rng.integers(1, 50, (changes, K)).astype(np.int32), np.zeros(0, np.int32),
                                 np.zeros(0, np.int32))
    ws = mb.Workspace(timeout_ms=20000)
    ws.set_grid(ctas, 0)
    assert_matches_oracle(run_update_device(ws, g, b), g, b)
    ws.close()
