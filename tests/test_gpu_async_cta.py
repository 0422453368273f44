"""The parts of the asynchronous near-far loop where sizes decide: rows at
the edges of a row record (three to nine edges), wavefronts that outgrow a
warp, a CTA's ring and its spill queue, and chains of single hops. Whole
numbers: every tree equals the oracle's."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mosp_b200 as mb  # noqa: E402
import oracle as orc  # noqa: E402
from gpu_util import assert_matches_oracle, dev, run_update_device  # noqa: E402


def csr(n, src, dst, K, rng, wmax=50):
    keep = src != dst
    keys = np.unique(src[keep].astype(np.int64) * n + dst[keep])
    row = np.searchsorted(keys, np.arange(n + 1) * np.int64(n)).astype(np.int32)
    return row, (keys % n).astype(np.int32), rng.integers(1, wmax + 1, (len(keys), K)).astype(np.int32)


def chain(n, fan, rng, K):
    """Vertex v to v + 1 .. v + fan: n - 1 hops in a row, rows of `fan` edges."""
    src = np.repeat(np.arange(n), fan)
    dst = src + np.tile(np.arange(1, fan + 1), n)
    ok = dst < n
    return csr(n, src[ok], dst[ok], K, rng)


def spread(n, fan, rng, K):
    """A tree of `fan` children per vertex plus n / 4 random edges: the
    wavefront grows from one entry past a warp, a ring and a CTA."""
    child = np.arange(1, n)
    src = np.concatenate([(child - 1) // fan, rng.integers(0, n, n // 4)])
    return csr(n, src, np.concatenate([child, rng.integers(0, n, n // 4)]), K, rng)


def from_scratch(ws, g, arrays, delta):
    row, col, w = arrays
    dg = mb.DeviceGraph.upload(ws, g)
    d = torch.empty(g.n, dtype=torch.int64, device="cuda")
    p = torch.empty(g.n, dtype=torch.int32, device="cuda")
    ws.sosp_from_scratch(g.n, g.m, dg.out_row, dg.out_col, dg.out_w[:g.m], 0, delta, int(w.max()), d, p)
    de, pe = orc.dijkstra(row, col, w, 0, 0)
    assert np.array_equal(d.cpu().numpy(), de) and np.array_equal(p.cpu().numpy(), pe)


@pytest.mark.parametrize("delta", [30, 10 ** 9])
@pytest.mark.parametrize("fan", [1, 2, 3, 4, 5, 8, 9])
def test_rows_around_a_record(fan, delta):
    """Average degrees on both sides of the row-record rule (3.5 edges per
    vertex), rows of one record, of one more edge and of several."""
    rng = np.random.default_rng(100 + fan)
    arrays = chain(3000, fan, rng, 2)
    g = mb.HostGraph.from_arrays(*arrays)
    ws = mb.Workspace(timeout_ms=20000)
    from_scratch(ws, g, arrays, delta)
    b = mb.HostBatch.generate(g, 200, seed=fan, wmax=50)
    assert_matches_oracle(run_update_device(ws, g, b), g, b)
    ws.close()


@pytest.mark.parametrize("ctas", [0, 1])
@pytest.mark.parametrize("n,fan,slots", [(33, 3, 0), (2000, 3, 0), (150000, 3, 0), (150000, 3, 2048),
                                         (150000, 2, 0), (60000, 30, 0)])
def test_wavefront_outgrows_warp_ring_and_cta(n, fan, slots, ctas):
    """One entry to tens of thousands within a phase, on the whole grid and on
    one CTA (whose ring then overflows into the spill queue; 2,048 slots:
    past it into the far pile)."""
    rng = np.random.default_rng(n + fan)
    arrays = spread(n, fan, rng, 1)
    g = mb.HostGraph.from_arrays(*arrays)
    ws = mb.Workspace(timeout_ms=20000)
    ws.set_async(True, slots)
    ws.set_grid(ctas, 0)
    for delta in (100, 10 ** 9):
        from_scratch(ws, g, arrays, delta)
    ws.close()


def test_bound_next_to_the_word():
    """A distance bound within 2^31 of what a packed word holds (the bulk
    loop runs) and just past that margin (the asynchronous loop runs)."""
    n = 3000
    rng = np.random.default_rng(7)
    row, col, _ = chain(n, 2, rng, 1)
    bits = 12  # 2^12 - 1 >= 3000 vertices
    top = (2 ** 64 - 1) >> bits
    for max_weight in (top // (n - 1), (top - 2 ** 31 - 1) // (n - 1)):
        w = rng.integers(1, 2 ** 31 - 1, (len(col), 1)).astype(np.int32)
        g = mb.HostGraph.from_arrays(row, col, w)
        ws = mb.Workspace(timeout_ms=20000)
        assert mb.choose_packing(n, max_weight)[0] == bits
        d, p = dev(np.zeros(n, np.int64)), dev(np.zeros(n, np.int32))
        dg = mb.DeviceGraph.upload(ws, g)
        ws.sosp_from_scratch(n, g.m, dg.out_row, dg.out_col, dg.out_w[:g.m], 0, 10 ** 11, max_weight, d, p)
        de, pe = orc.dijkstra(row, col, w, 0, 0)
        assert np.array_equal(d.cpu().numpy(), de) and np.array_equal(p.cpu().numpy(), pe)
        ws.close()
