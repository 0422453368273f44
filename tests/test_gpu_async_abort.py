"""A launch of the asynchronous loop that runs out of time: the call returns
its timeout within seconds, whatever its warps were at (most of them wait for mail
that never comes), and the workspace is as good as new."""
import time

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
import oracle as orc  # noqa: E402


def chain(n, fan):
    """Vertex v to v + 1 .. v + fan, all of weight 1: n - 1 hops in a row."""
    src = np.repeat(np.arange(n), fan)
    dst = src + np.tile(np.arange(1, fan + 1), n)
    ok = dst < n
    row = np.concatenate([[0], np.cumsum(np.bincount(src[ok], minlength=n))]).astype(np.int32)
    return row, dst[ok].astype(np.int32), np.ones((int(ok.sum()), 1), np.int32)


def limit_ms(ws, ms):
    mb.check(mb.lib().mosp_workspace_set_timeout_ms(ws._h, ms))


@pytest.mark.parametrize("fan", [1, 4, 6])
def test_timeout_while_warps_wait_for_mail(fan):
    """One phase of several hundred thousand hops (rows of one edge, of a full
    row record, and without records): at the deadline one warp of the grid has
    work and the others wait, most of which were never sent anything."""
    n = 300000 * fan
    row, col, w = chain(n, fan)
    g = mb.HostGraph.from_arrays(row, col, w)
    ws = mb.Workspace(timeout_ms=20000)
    dg = mb.DeviceGraph.upload(ws, g)
    d = torch.empty(n, dtype=torch.int64, device="cuda")
    p = torch.empty(n, dtype=torch.int32, device="cuda")
    args = (n, g.m, dg.out_row, dg.out_col, dg.out_w[:g.m], 0, 10 ** 9, 1, d, p)
    de, pe = orc.dijkstra(row, col, w, 0, 0)
    for limit in (4, 9, 20):
        limit_ms(ws, limit)
        t0 = time.perf_counter()
        with pytest.raises(mb.MospError) as e:
            ws.sosp_from_scratch(*args)
        assert e.value.status == mb.ERR_TIMEOUT
        assert time.perf_counter() - t0 < limit / 1000 + 5.0
        limit_ms(ws, 20000)
        ws.sosp_from_scratch(*args)
        assert np.array_equal(d.cpu().numpy(), de) and np.array_equal(p.cpu().numpy(), pe)
    ws.close()
