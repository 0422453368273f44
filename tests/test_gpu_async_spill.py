"""Which parts of the asynchronous loop a launch went through, by its own
counts: chains stay with their CTAs, wavefronts past a CTA's ring go through
the spill queue, and with a queue that is too small through the far pile."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
import oracle as orc  # noqa: E402


def graph(n, fan, rng):
    """Children fan v + 1 .. fan v + fan (fan 1: a chain), and n / 4 random
    edges where the tree branches."""
    child = np.arange(1, n)
    more = rng.integers(0, n, (2, n // 4 if fan > 1 else 0))
    src = np.concatenate([(child - 1) // fan, more[0]])
    keys = np.unique(src * np.int64(n) + np.concatenate([child, more[1]]))
    keys = keys[keys // n != keys % n]
    row = np.searchsorted(keys, np.arange(n + 1) * np.int64(n)).astype(np.int32)
    col = (keys % n).astype(np.int32)
    return row, col, rng.integers(1, 51, (len(col), 1)).astype(np.int32)


@pytest.mark.parametrize("fan,ctas,slots", [(1, 0, 0), (3, 1, 0), (3, 0, 0), (3, 1, 2048), (30, 0, 0)])
def test_route_of_a_wavefront(fan, ctas, slots):
    n = 20000 if fan == 1 else 150000
    row, col, w = graph(n, fan, np.random.default_rng(fan))
    g = mb.HostGraph.from_arrays(row, col, w)
    ws = mb.Workspace(timeout_ms=20000)
    ws.set_async(True, slots)
    ws.set_grid(ctas, 0)
    dg = mb.DeviceGraph.upload(ws, g)
    d = torch.empty(n, dtype=torch.int64, device="cuda")
    p = torch.empty(n, dtype=torch.int32, device="cuda")
    st = ws.sosp_from_scratch(n, g.m, dg.out_row, dg.out_col, dg.out_w[:g.m], 0, 10 ** 9, 50, d, p)
    de, pe = orc.dijkstra(row, col, w, 0, 0)
    assert np.array_equal(d.cpu().numpy(), de) and np.array_equal(p.cpu().numpy(), pe)
    assert st.iterations == st.epochs  # (the bulk loop counts its iterations apart)
    prof = ws.loop_profile(0, True)
    assert 0 < prof["local_rounds"] <= prof["warp_rounds"]
    if fan == 1:
        assert prof["queue_entries"] == 0 and prof["local_rounds"] == prof["warp_rounds"]
        assert prof["phases"] == 1
    else:
        # (a phase of everything: 10^9 is past every distance)
        assert prof["queue_entries"] > 0 and prof["local_rounds"] < prof["warp_rounds"]
        assert prof["phases"] > 1 if slots else prof["phases"] == 1
    ws.close()
