"""Step 1 on parallel edges that lie apart in a long row: the walk from a
group's first occurrence to the last one that it touches takes 16 heads at a
time. Occurrences at the edges of such a block, rows that end inside one, and
edges that go, stay and take weights within one. Equal to the host
application edge for edge."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
from gpu_util import dev  # noqa: E402
from test_gpu_apply_fused import check  # noqa: E402


@pytest.mark.parametrize("gaps", [[1, 1, 1], [15, 1, 15], [16, 16, 16], [17, 15, 1], [14, 2, 33], [31, 65, 400]])
@pytest.mark.parametrize("behind", [0, 1, 15, 40])
def test_occurrences_apart(gaps, behind):
    rng = np.random.default_rng(sum(gaps) + behind)
    n, K = 700, 3
    at = np.concatenate([[5], 5 + np.cumsum(gaps)])  # occurrences of head 1 in each row
    long_row = rng.integers(2, n, at[-1] + 1 + behind)
    long_row[at] = 1
    degrees = np.array([len(long_row)] * 12 + [1] * (n - 13) + [len(long_row)])
    col = np.concatenate([long_row if d > 1 else [1] for d in degrees]).astype(np.int32)
    row = np.concatenate([[0], np.cumsum(degrees)]).astype(np.int32)
    w = rng.integers(1, 1000, (len(col), K)).astype(np.int32)
    # deletions and insertions of (u, 1): 0 to 5 of one and 0 to 2 of the other
    pairs = [(0, 1), (1, 0), (1, 1), (2, 0), (2, 1), (3, 1), (3, 2), (4, 0), (4, 1), (5, 1), (0, 2), (2, 2), (3, 1)]
    rows = list(range(12)) + [n - 1]
    del_from = np.concatenate([[u] * d for u, (d, _) in zip(rows, pairs)]).astype(np.int32)
    ins_from = np.concatenate([[u] * i for u, (_, i) in zip(rows, pairs)]).astype(np.int32)
    check(row, col, w, {"ins_from": ins_from, "ins_to": np.ones_like(ins_from),
                        "ins_w": rng.integers(1, 900, (len(ins_from), K)).astype(np.int32),
                        "del_from": del_from, "del_to": np.ones_like(del_from)})


def test_a_million_edges_apart():
    """Head by head the walk takes 113 ms (and 90 in the sorted form)."""
    m, K, n = 1000000, 1, 1000
    head = torch.randint(2, n, (m,), dtype=torch.int32, device="cuda")
    head[0] = head[m - 1] = 1
    row = dev(np.where(np.arange(n + 1) > 0, m, 0).astype(np.int32))
    w = torch.ones(m, dtype=torch.int32, device="cuda")
    gone = [dev(np.array(x, np.int32)) for x in ([0, 0], [1, 1])]
    none = torch.zeros(0, dtype=torch.int32, device="cuda")
    new = [torch.zeros(x, dtype=torch.int32, device="cuda") for x in (n + 1, m, m, 1)]
    ws = mb.Workspace(timeout_ms=20000)
    times = []
    for _ in range(3):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        new_m, _, _ = ws.apply_batch_device(n, K, m, row, head, w, none, none, none, *gone, *new)
        end.record()
        torch.cuda.synchronize()
        times.append(start.elapsed_time(end))
    ws.close()
    assert new_m == m - 2 and torch.equal(new[1][:new_m], head[1:m - 1])
    assert min(times) < 60
