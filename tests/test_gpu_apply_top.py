"""Step 1 at the top of the accepted range: the graph and its insertions have
2^31 - 1 edges, so positions just past a row's or a piece's end do not fit 32
signed bits. Equal to the host application: the changes touch the last edges,
which make a small host graph, and all others only move."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
from gpu_util import dev  # noqa: E402

TOP = 2 ** 31 - 1


def equal(a, b):
    step = 1 << 28
    return len(a) == len(b) and all(torch.equal(a[i:i + step], b[i:i + step]) for i in range(0, len(a), step))


@pytest.mark.parametrize("slack", [0, 33])
@pytest.mark.parametrize("lengths", [[], [100, 1, 0, 31, 70, 17, 2, 16, 40, 3]])
def test_two_billion_edges(lengths, slack):
    """One row of everything, and short rows behind it."""
    if torch.cuda.mem_get_info()[0] < 50 << 30:
        pytest.skip("needs 50 GB of device memory")
    rng = np.random.default_rng(len(lengths) + slack)
    n, n_ins, n_del = 1000, 12, 6
    degrees = np.array([50] + lengths + [0] * (n - 1 - len(lengths)))
    rows = np.flatnonzero(degrees)
    # the tails of the rows: heads 500 .. 999, the rest of row 0 has others
    col = np.concatenate([rng.choice(np.arange(500, n), d, replace=False) for d in degrees]).astype(np.int32)
    row = np.concatenate([[0], np.cumsum(degrees)]).astype(np.int32)
    w = rng.integers(1, 1000, (len(col), 1)).astype(np.int32)
    tail = np.repeat(np.arange(n), degrees)
    old = np.concatenate([rng.integers(0, len(col), 3), [len(col) - 1]])
    ins_from = np.concatenate([tail[old], rng.choice(rows, 6), rows[[-1, -1]]])
    ins_to = np.concatenate([col[old], rng.integers(500, n, n_ins - 4)])
    gone = np.concatenate([rng.integers(0, len(col), n_del - 2), [len(col) - 2, 0]])
    ins_w = rng.integers(1, 900, (n_ins, 1)).astype(np.int32)
    g = mb.HostGraph.from_arrays(row, col, w)
    b = mb.HostBatch.from_arrays(1, ins_from, ins_to, ins_w, tail[gone], col[gone])
    er, ec, ew = mb.apply_batch(g, b).arrays()
    rest = TOP - slack - n_ins - len(col)
    m = rest + len(col)
    big_col = torch.empty(m, dtype=torch.int32, device="cuda")
    big_col[:rest].random_(0, 500)
    big_col[rest:] = dev(col)
    big_w = torch.empty(m, dtype=torch.int32, device="cuda")
    big_w[:rest].random_(1, 1000)
    big_w[rest:] = dev(w.reshape(-1))
    big_row = dev((row.astype(np.int64) + np.where(np.arange(n + 1) > 0, rest, 0)).astype(np.int32))
    new_row, mask = dev(np.zeros(n + 1, np.int32)), dev(np.zeros(n_ins, np.int32))
    new_col = torch.zeros(m + n_ins, dtype=torch.int32, device="cuda")
    new_w = torch.zeros(m + n_ins, dtype=torch.int32, device="cuda")
    ws = mb.Workspace(timeout_ms=20000)
    i32 = lambda x: dev(np.ascontiguousarray(x, np.int32))  # noqa: E731
    nm, most, total = ws.apply_batch_device(n, 1, m, big_row, big_col, big_w, i32(ins_from), i32(ins_to),
                                            i32(ins_w.reshape(-1)), i32(tail[gone]), i32(col[gone]), new_row,
                                            new_col, new_w, mask)
    ws.close()
    assert nm == rest + len(ec)
    assert np.array_equal(new_row.cpu().numpy(), er.astype(np.int64) + np.where(np.arange(n + 1) > 0, rest, 0))
    assert np.array_equal(new_col[rest:nm].cpu().numpy(), ec)
    assert np.array_equal(new_w[rest:nm].cpu().numpy(), ew.reshape(-1))
    assert equal(new_col[:rest], big_col[:rest]) and equal(new_w[:rest], big_w[:rest])
    assert np.array_equal(mask.cpu().numpy().view(np.uint32), b.arrays()["mask"])
    assert total[0] == sum(int(big_w[i:i + (1 << 28)].sum(dtype=torch.int64)) for i in range(0, m, 1 << 28))
    del big_col, big_w, new_col, new_w
    torch.cuda.empty_cache()
