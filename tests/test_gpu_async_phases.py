"""Hundreds of short phases in one launch: warps go idle and are sent mail or
woken at each end. A wake-up that is lost ends in a timeout, mail read too
early in a wrong tree."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
import oracle as orc  # noqa: E402


@pytest.mark.parametrize("ctas", [0, 1, 3])
@pytest.mark.parametrize("width", [12, 40])
def test_many_short_phases(width, ctas):
    """A band of `width` vertices a step, three edges each into the next step
    (wavefronts of more than a warp's eight entries), a few steps per phase."""
    steps = 400
    n = width * steps
    rng = np.random.default_rng(width)
    v = np.repeat(np.arange(n - width), 3)
    to = (v // width + 1) * width + (v % width + np.tile([0, 1, 5], n - width)) % width
    first = np.arange(1, width)
    keys = np.unique(np.concatenate([v * np.int64(n) + to, first]))
    row = np.searchsorted(keys, np.arange(n + 1) * np.int64(n)).astype(np.int32)
    col = (keys % n).astype(np.int32)
    w = rng.integers(1, 11, (len(col), 1)).astype(np.int32)
    g = mb.HostGraph.from_arrays(row, col, w)
    de, pe = orc.dijkstra(row, col, w, 0, 0)
    ws = mb.Workspace(timeout_ms=5000)
    ws.set_grid(ctas, 0)
    dg = mb.DeviceGraph.upload(ws, g)
    d = torch.empty(n, dtype=torch.int64, device="cuda")
    p = torch.empty(n, dtype=torch.int32, device="cuda")
    for delta in (3, 10, 30) * 5:
        ws.sosp_from_scratch(n, g.m, dg.out_row, dg.out_col, dg.out_w[:g.m], 0, delta, 10, d, p)
        assert np.array_equal(d.cpu().numpy(), de) and np.array_equal(p.cpu().numpy(), pe)
        assert ws.loop_profile(0, True)["phases"] > 10
    ws.close()
