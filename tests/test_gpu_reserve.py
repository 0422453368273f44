"""What a workspace allocates once its user has reserved it: nothing, for any
graph within the reserved size (an allocation or its release waits for the
whole device, also for launches of other streams)."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
from gpu_util import dev  # noqa: E402


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def rows_of(n, m):
    """n rows of m edges in all, as equal as they get."""
    return dev((np.arange(n + 1, dtype=np.int64) * m // n).astype(np.int32))


def device_graph(n, m, K, gen, wmax=100):
    """Room for K weights on each of m random edges of n vertices, and for the
    arrays of the device graph."""
    col = torch.randint(0, n, (m,), generator=gen, device="cuda", dtype=torch.int32)
    w = torch.randint(1, wmax + 1, (m * K,), generator=gen, device="cuda", dtype=torch.int32)
    return col, w, [torch.zeros(x, dtype=torch.int32, device="cuda") for x in (m * K, n + 1, m, m * K)]


def test_builds_of_a_growing_graph():
    """A graph that gains edges from build to build: nothing is allocated after
    a reservation, and without one only a few times (20 builds, 40 MB of ranks,
    each 4 MB more than the last)."""
    n, K, m0, step = 100000, 1, 10 ** 7, 10 ** 6
    gen = torch.Generator(device="cuda").manual_seed(1)
    col, w, out = device_graph(n, m0 + 19 * step, K, gen)
    for reserved in (True, False):
        ws = mb.Workspace(timeout_ms=20000)
        if reserved:
            mb.check(mb.lib().mosp_workspace_reserve_graph(ws._h, n, m0 + 19 * step, K))
        seen = {free_bytes()} if reserved else set()
        for i in range(20):
            m = m0 + i * step
            row = rows_of(n, m)
            ws.build_device_graph(n, m, K, row, col, w, *out)
            assert int(out[1][n]) == m
            seen.add(free_bytes())
        # (growth by half again: 10.1, 15.2, 22.7 and 34.1 million entries)
        assert len(seen) == (1 if reserved else 1 + math.ceil(math.log((n + m) / (n + m0), 1.5)))
        ws.close()


def update_of(ws, n, m, K, max_weight, gen):
    """K trees of a random graph, then an update without changes, which leaves
    them."""
    col, w, (out_w, in_row, in_col, in_w) = device_graph(n, m, K, gen)
    row = rows_of(n, m)
    dist = torch.zeros(K * n, dtype=torch.int64, device="cuda")
    par = torch.zeros(K * n, dtype=torch.int32, device="cuda")
    cd, cp = torch.zeros(n, dtype=torch.int64, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
    none = torch.zeros(1, dtype=torch.int32, device="cuda")
    ws.build_device_graph(n, m, K, row, col, w, out_w, in_row, in_col, in_w)
    for k in range(K):
        ws.sosp_from_scratch(n, m, row, col, out_w[k * m:], 0, 100, max_weight, dist[k * n:], par[k * n:])
    want = dist.clone(), par.clone()
    ws.update_device(n, m, K, row, col, out_w, in_row, in_col, in_w, none, none, [0] * (K + 1), none, 0, 0,
                     [100] * K, [max_weight] * K, None, dist, par, cd, cp)
    assert torch.equal(dist, want[0]) and torch.equal(par, want[1])


@pytest.mark.parametrize("max_weight", [100, 1 << 30])
def test_sparser_graph_than_reserved(max_weight):
    """Reserved for 5 edges per vertex, where the loop takes no row records;
    updates of graphs with 4 and 2 (records), with parents beside the distances
    and recovered after them."""
    n, m, K = 10 ** 6, 5 * 10 ** 6, 2
    gen = torch.Generator(device="cuda").manual_seed(2)
    update_of(mb.Workspace(timeout_ms=20000), 1000, 3000, K, max_weight, gen)  # kernels and caches are loaded
    ws = mb.Workspace(timeout_ms=20000)
    mb.check(mb.lib().mosp_workspace_reserve_graph(ws._h, n, m, K))
    for edges in (m, 4 * n, 2 * n):
        pool = torch.zeros(1 << 27, dtype=torch.int64, device="cuda")
        del pool  # (kept by torch, which takes the graph and the trees from it)
        before = free_bytes()
        update_of(ws, n, edges, K, max_weight, gen)
        assert free_bytes() == before
    ws.close()
