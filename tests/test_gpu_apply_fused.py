"""The one-launch batch application where its routes part: touched rows at the
edges of a lane's, a piece's and several pieces' length, repeated edges,
several deletions and insertions of one edge, rows whose removed edges span
copy chunks, numbers of objectives that do and do not divide a warp. Equal to the host application
edge for edge."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
from gpu_util import dev  # noqa: E402


def check(row, col, w, batch):
    n, m, K = len(row) - 1, len(col), w.shape[1]
    g = mb.HostGraph.from_arrays(row, col, w)
    b = mb.HostBatch.from_arrays(K, batch["ins_from"], batch["ins_to"], batch["ins_w"], batch["del_from"],
                                 batch["del_to"])
    er, ec, ew = mb.apply_batch(g, b).arrays()
    mask = b.arrays()["mask"]
    n_ins = len(batch["ins_from"])
    cap = m + n_ins
    new = [dev(np.zeros(max(x, 1), np.int32)) for x in (n + 1, cap, cap * K, n_ins)]
    ws = mb.Workspace(timeout_ms=20000)
    t = {k: dev(np.ascontiguousarray(v, np.int32)) for k, v in batch.items()}
    args = (n, K, m, dev(row), dev(col), dev(w.reshape(-1)), t["ins_from"], t["ins_to"], t["ins_w"], t["del_from"],
            t["del_to"], *new)
    for _ in range(2):
        nm, most, total = ws.apply_batch_device(*args[:11], new[0], new[1], new[2], new[3])
        assert nm == len(ec)
        assert np.array_equal(new[0].cpu().numpy(), er)
        assert np.array_equal(new[1].cpu().numpy()[:nm], ec)
        assert np.array_equal(new[2].cpu().numpy()[:nm * K].reshape(nm, K), ew)
        assert np.array_equal(new[3].cpu().numpy()[:n_ins].view(np.uint32), mask)
        for k in range(K):
            assert total[k] == int(w[:, k].sum())
            assert most[k] == max(1, int(w[:, k].max()) if m else 1,
                                  int(batch["ins_w"][:, k].max()) if n_ins else 1)
    ws.close()


def rows_of(degrees, n, rng, repeats):
    """Rows of the given lengths; every `repeats`-th edge repeats an earlier
    head of its row."""
    cols = []
    for d in degrees:
        c = rng.integers(0, n, d)
        if repeats:
            at = np.arange(repeats, d, repeats)
            c[at] = c[rng.integers(0, np.maximum(at, 1))] if len(at) else c[at]
        cols.append(c)
    row = np.concatenate([[0], np.cumsum(degrees)]).astype(np.int32)
    return row, np.concatenate(cols).astype(np.int32)


def changes(row, col, K, rng, n_ins, n_del, again):
    n, m = len(row) - 1, len(col)
    tail = np.repeat(np.arange(n), np.diff(row))
    pick = rng.integers(0, m, n_del)
    old = rng.integers(0, m, n_ins // 2)
    ins_from = np.concatenate([tail[old], rng.integers(0, n, n_ins - len(old))])
    ins_to = np.concatenate([col[old], rng.integers(0, n, n_ins - len(old))])
    if again:  # several changes of the same edge
        ins_from[1::3], ins_to[1::3] = ins_from[0], ins_to[0]
        pick[::4] = pick[0] if n_del else pick[::4]
    order = rng.permutation(n_ins)
    return {"ins_from": ins_from[order], "ins_to": ins_to[order], "ins_w": rng.integers(1, 900, (n_ins, K)),
            "del_from": tail[pick], "del_to": col[pick]}


@pytest.mark.parametrize("repeats", [0, 3])
@pytest.mark.parametrize("K", [1, 2, 3, 5, 7, 17, 32])
def test_row_lengths_and_objectives(K, repeats):
    rng = np.random.default_rng(10 * K + repeats)
    degrees = [0, 1, 15, 16, 17, 31, 32, 33, 63, 64, 65, 128, 129, 5000, 0, 3] + [2] * 500
    n = len(degrees)
    row, col = rows_of(degrees, n, rng, repeats)
    w = rng.integers(1, 1000, (len(col), K)).astype(np.int32)
    check(row, col, w, changes(row, col, K, rng, 900, 900, repeats > 0))


@pytest.mark.parametrize("n_ins,n_del", [(0, 1), (1, 0), (40000, 0), (0, 40000), (20000, 20000)])
def test_one_row_takes_the_batch(n_ins, n_del):
    """A row of 50,000 edges with most of the changes: removed edges in every
    copy chunk, thousands of appended ones."""
    rng = np.random.default_rng(n_ins + 2 * n_del)
    n = 70000
    row, col = rows_of([50000] + [1] * (n - 1), n, rng, 0)
    w = rng.integers(1, 1000, (len(col), 2)).astype(np.int32)
    b = changes(row, col, 2, rng, n_ins, n_del, False)
    b["ins_from"][: n_ins * 3 // 4] = 0
    check(row, col, w, b)


def test_no_edges():
    check(np.zeros(6, np.int32), np.zeros(0, np.int32), np.zeros((0, 2), np.int32),
          {"ins_from": np.array([4, 0, 4]), "ins_to": np.array([1, 2, 1]),
           "ins_w": np.array([[3, 4], [5, 6], [7, 8]]), "del_from": np.array([2]), "del_to": np.array([3])})


@pytest.mark.parametrize("every", [1, 2, 5])
@pytest.mark.parametrize("last", [0, 1, 31])
@pytest.mark.parametrize("degrees", [[1] * 96, [32] * 4, [0, 0, 0, 16] * 10, [31, 1, 0, 33, 0, 0, 63, 65], [130, 0, 0]])
def test_moves_within_blocks_of_edges(degrees, last, every):
    """Appended, removed and overwritten edges at every place of the copy's
    blocks of 32: an append before each edge of a block, rows that end at a
    block's end, several appends at one place (also through empty rows), a
    last block of 1, 31 and 32 edges."""
    rng = np.random.default_rng(1000 * every + 10 * last + len(degrees))
    degrees = degrees + [last]
    n, K = len(degrees) + 200, 3
    row, col = rows_of(degrees + [0] * 200, n, rng, 0)
    w = rng.integers(1, 1000, (len(col), K)).astype(np.int32)
    tail = np.repeat(np.arange(n), np.diff(row))
    rows = np.repeat(np.arange(0, len(degrees), every), 1 + (every == 5))  # one or two per row
    take = np.arange(0, len(col), 7)
    batch = {"ins_from": np.concatenate([rows, tail[take + (take + 1 < len(col))]]),
             "ins_to": np.concatenate([rng.integers(0, n, len(rows)), col[take + (take + 1 < len(col))]]),
             "del_from": tail[take], "del_to": col[take]}
    batch["ins_w"] = rng.integers(1, 900, (len(batch["ins_from"]), K))
    check(row, col, w, batch)
