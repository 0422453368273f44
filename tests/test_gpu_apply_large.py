"""Batches of about 2^18 changes on a graph with fewer vertices than the
batch has entries: the scans over the batch are the longest ones of Step 1.
Equal to the host application edge for edge."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
from gpu_util import dev  # noqa: E402


@pytest.mark.parametrize("changes", [262144, 262146, 400000])
def test_more_changes_than_vertices(changes):
    rng = np.random.default_rng(changes)
    n, m, K = 60000, 240000, 2
    row = np.arange(0, m + 1, 4).astype(np.int32)
    col = rng.integers(0, n, m).astype(np.int32)
    w = rng.integers(1, 1000, (m, K)).astype(np.int32)
    n_ins = changes // 2
    pick, old = rng.integers(0, m, changes - n_ins), rng.integers(0, m, n_ins // 2)
    b = {"ins_from": np.concatenate([old // 4, rng.integers(0, n, n_ins - len(old))]),
         "ins_to": np.concatenate([col[old], rng.integers(0, n, n_ins - len(old))]),
         "ins_w": rng.integers(1, 900, (n_ins, K)), "del_from": pick // 4, "del_to": col[pick]}
    hb = mb.HostBatch.from_arrays(K, b["ins_from"], b["ins_to"], b["ins_w"], b["del_from"], b["del_to"])
    er, ec, ew = mb.apply_batch(mb.HostGraph.from_arrays(row, col, w), hb).arrays()
    t = {k: dev(np.ascontiguousarray(v, np.int32)) for k, v in b.items()}
    new = [dev(np.zeros(x, np.int32)) for x in (n + 1, m + n_ins, (m + n_ins) * K, n_ins)]
    ws = mb.Workspace(timeout_ms=20000)
    nm, _, _ = ws.apply_batch_device(n, K, m, dev(row), dev(col), dev(w.reshape(-1)), t["ins_from"], t["ins_to"],
                                     t["ins_w"], t["del_from"], t["del_to"], *new)
    ws.close()
    assert nm == len(ec) and np.array_equal(new[0].cpu().numpy(), er)
    assert np.array_equal(new[1].cpu().numpy()[:nm], ec)
    assert np.array_equal(new[2].cpu().numpy()[:nm * K].reshape(nm, K), ew)
    assert np.array_equal(new[3].cpu().numpy().view(np.uint32), hb.arrays()["mask"])
