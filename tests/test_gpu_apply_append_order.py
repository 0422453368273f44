"""Step 1 with many edges appended to few rows: a row that takes more than one
in sixteen of a batch's insertions orders them by a bit per insertion, others
by their list. Counts at that line, batches below and above the size from which
there are bits, last insertions at the edges of a word and of four. Equal to the
host application edge for edge."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
from gpu_util import dev  # noqa: E402
from test_gpu_apply_fused import check  # noqa: E402


@pytest.mark.parametrize("n_ins", [8192, 8193, 8224, 10000, 10113])
@pytest.mark.parametrize("share", ["one", "line", "all rows", "last row"])
def test_order_of_appended_edges(n_ins, share):
    rng = np.random.default_rng(n_ins)
    n, K = 12000, 2
    degrees = rng.integers(0, 5, n)
    row = np.concatenate([[0], np.cumsum(degrees)]).astype(np.int32)
    col = rng.integers(0, n, row[-1]).astype(np.int32)
    w = rng.integers(1, 1000, (len(col), K)).astype(np.int32)
    line = n_ins // 16
    if share == "one":
        ins_from = np.full(n_ins, 77)
    elif share == "line":  # rows just above and at the line; the rest everywhere
        ins_from = np.concatenate([np.repeat([3, 900, n - 1], line + 1), np.repeat([5, 901, n - 3], line),
                                   rng.integers(0, n, n_ins - 3 * (2 * line + 1))])
    elif share == "all rows":  # fifteen rows above the line
        ins_from = np.arange(n_ins) % 15 + 40
    else:
        ins_from = np.where(np.arange(n_ins) % 3 == 0, 9, n - 1)
    ins_from = rng.permutation(ins_from).astype(np.int32)
    # distinct heads but for a few that repeat an insertion or an edge
    ins_to = rng.permutation(n)[:n_ins].astype(np.int32)
    ins_to[rng.integers(0, n_ins, 50)] = ins_to[rng.integers(0, n_ins, 50)]
    pick = np.flatnonzero(degrees[ins_from] > 0)[:40]
    ins_to[pick] = col[row[ins_from[pick]]]
    gone = rng.integers(0, len(col), 60)
    tail = np.repeat(np.arange(n), degrees).astype(np.int32)
    check(row, col, w, {"ins_from": ins_from, "ins_to": ins_to,
                        "ins_w": rng.integers(1, 900, (n_ins, K)).astype(np.int32),
                        "del_from": tail[gone], "del_to": col[gone]})


def test_a_batch_into_one_row():
    """200,000 edges appended to one row: list against list takes 8.8 ms (6.3
    in the sorted form)."""
    n, n_ins, K = 200001, 200000, 1
    i32 = lambda x: dev(np.ascontiguousarray(x, np.int32))  # noqa: E731
    none = torch.zeros(0, dtype=torch.int32, device="cuda")
    order = np.random.default_rng(3).permutation(n_ins)
    ins = [i32(np.full(n_ins, 7)), i32(order), i32(np.ones(n_ins))]
    one = [i32(np.where(np.arange(n + 1) > 5, 1, 0)), i32([3]), i32([9])]
    new = [torch.zeros(x, dtype=torch.int32, device="cuda") for x in (n + 1, n_ins + 1, n_ins + 1, n_ins)]
    ws = mb.Workspace(timeout_ms=20000)
    times = []
    for _ in range(4):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        new_m, _, _ = ws.apply_batch_device(n, K, 1, *one, *ins, none, none, *new)
        end.record()
        torch.cuda.synchronize()
        times.append(start.elapsed_time(end))
    ws.close()
    assert new_m == n_ins + 1 and np.array_equal(new[1].cpu().numpy(), np.concatenate([[3], order]))
    assert min(times) < 4
