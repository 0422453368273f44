"""Workspaces on a device with little memory left: the arrays that only make
calls faster are left out or given back, and what has room without them runs,
with the same results."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
import oracle as orc  # noqa: E402
from gpu_util import dev  # noqa: E402

MB = 1 << 20


class Full:
    """All but `left` bytes of the device's memory taken."""

    def __init__(self, left):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        size = torch.cuda.mem_get_info()[0] - left
        self.hold = torch.empty(size, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *_):
        del self.hold
        torch.cuda.empty_cache()


def test_update_with_room_for_the_bulk_loop_only():
    """A grid of 1M vertices, K = 3. Without records, far copies and spill
    queue: 32 bytes of lists and 48 of near lists per vertex and objective, 8
    n (K + 1) of the combined graph, and 24 MB for the rest."""
    side, K = 1000, 3
    n = side * side
    rng = np.random.default_rng(3)
    v = np.arange(n)
    right, down = v[v % side < side - 1], v[: n - side]
    a, b = np.concatenate([right, down]), np.concatenate([right + 1, down + side])
    keys = np.sort(np.concatenate([a * np.int64(n) + b, b * np.int64(n) + a]))
    row = np.searchsorted(keys, np.arange(n + 1) * np.int64(n)).astype(np.int32)
    col, m = (keys % n).astype(np.int32), len(keys)
    w = rng.integers(1, 100, (m, K)).astype(np.int32)
    # the trees of other weights on some edges, which the batch sets right
    w0 = w.copy()
    edge = rng.choice(m, 2000, replace=False)
    w0[edge] = rng.integers(1, 100, (len(edge), K))
    tail = np.repeat(v, np.diff(row)).astype(np.int32)
    init = [orc.dijkstra(row, col, w0, k, 0) for k in range(K)]
    want = [orc.dijkstra(row, col, w, k, 0) for k in range(K)]
    d_row, d_col, d_w = dev(row), dev(col), dev(w.reshape(-1))
    out_w, in_row, in_col, in_w = [torch.zeros(x, dtype=torch.int32, device="cuda") for x in (m * K, n + 1, m, m * K)]
    dist, par = dev(np.stack([x[0] for x in init])), dev(np.stack([x[1] for x in init]))
    cd, cp = torch.zeros(n, dtype=torch.int64, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
    ch_from, ch_to = dev(np.tile(tail[edge], K)), dev(np.tile(col[edge], K))
    heads = dev(col[edge])
    first = mb.Workspace(timeout_ms=20000)  # kernels are loaded before the device is full
    first.build_device_graph(n, m, K, d_row, d_col, d_w, out_w, in_row, in_col, in_w)
    first.close()
    d, p = torch.empty_like(dist), torch.empty_like(par)
    with Full((32 + 48) * n * K + 8 * n * (K + 1) + 24 * MB):
        ws = mb.Workspace(timeout_ms=20000)
        for _ in range(2):
            d.copy_(dist)
            p.copy_(par)
            ws.update_device(n, m, K, d_row, d_col, out_w, in_row, in_col, in_w, ch_from, ch_to,
                             [len(edge) * k for k in range(K + 1)], heads, len(edge), 0, [300] * K, [100] * K, None,
                             d, p, cd, cp)
            for k in range(K):
                assert np.array_equal(d[k].cpu().numpy(), want[k][0]) and np.array_equal(p[k].cpu().numpy(), want[k][1])
        ws.close()


@pytest.mark.parametrize("K", [1, 3])
def test_build_without_room_for_ranks(K):
    """16M edges, whose ranks take 64 MB, with 24 MB left: the same reverse
    rows as with room (in-edges of a vertex in any order)."""
    n, m = 200000, 16 * 10 ** 6
    gen = torch.Generator(device="cuda").manual_seed(K)
    col = torch.randint(0, n, (m,), generator=gen, device="cuda", dtype=torch.int32)
    w = torch.randint(1, 100, (m * K,), generator=gen, device="cuda", dtype=torch.int32)
    row = dev((np.arange(n + 1, dtype=np.int64) * m // n).astype(np.int32))
    outs = [torch.zeros(x, dtype=torch.int32, device="cuda") for x in (m * K, n + 1, m, m * K)]
    out_w, in_row, in_col, in_w = outs

    def build(ws):
        for x in outs:
            x.zero_()
        ws.build_device_graph(n, m, K, row, col, w, out_w, in_row, in_col, in_w)

    def result():
        key = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.diff(in_row).long()) * n + in_col
        for k in range(K):
            key = key * 100 + in_w[k * m:(k + 1) * m]
        return torch.sort(key)[0], in_row.clone(), out_w.clone()

    ws = mb.Workspace(timeout_ms=20000)
    build(ws)
    want = result()
    ws.close()
    ws = mb.Workspace(timeout_ms=20000)
    with Full(24 * MB):
        build(ws)
        build(ws)
    assert all(torch.equal(a, b) for a, b in zip(result(), want))
    build(ws)  # with room again
    assert all(torch.equal(a, b) for a, b in zip(result(), want))
    ws.close()


def test_bulk_loop_allocates_nothing_for_the_other():
    """set_async(False): 32 bytes of lists per vertex and objective."""
    n, m, K = 2 * 10 ** 6, 2 * 10 ** 6, 4
    held = []
    for on in (True, False):
        torch.cuda.synchronize()
        ws = mb.Workspace(timeout_ms=20000)
        ws.set_async(on)
        before = torch.cuda.mem_get_info()[0]
        mb.check(mb.lib().mosp_workspace_reserve_graph(ws._h, n, m, K))
        held.append(before - torch.cuda.mem_get_info()[0])
        ws.close()
    # far copies 16 and records 32 bytes, spill queue 8 n (K + 1)
    assert abs(held[0] - held[1] - ((16 + 32) * n * K + 8 * n * (K + 1))) <= 8 * MB
