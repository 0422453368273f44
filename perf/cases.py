"""Timed cases of the MOSP update path.

Every case is one pass through the public Python binding (`mosp_b200`) on a
seeded synthetic graph: a road network (a grid with missing streets and a few
diagonal shortcuts, or a disjoint union of several) or a power-law R-MAT
graph, both as CSR with K weights per edge, and a batch of changed edges.

kinds
  update    mosp_update_device: the K tree updates, the combined graph and its
            tree, on a graph and trees that stay on the GPU
  step      mosp_build_device_graph, mosp_update_device and mosp_path_costs:
            all that follows the application of a batch to a resident graph
  apply     mosp_apply_batch_device: the application itself
  scratch   mosp_sosp_from_scratch: one objective's tree of a new graph
  combined  mosp_combined_sosp: the combined tree of given trees, as after a
            change of the preferences
  host      mosp_update_host: the whole update from host buffers

An update works in place on the trees, so a pass of `update` or `step` first
copies the trees of the unchanged graph into the working ones, as a program
does that tries several batches against one state of the network.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "mosp-cuda_b200"))

import mosp_b200 as mb  # noqa: E402

DEV = "cuda"


def _road(kind, rows, cols, K, changes, mode, instances=1, wmax=100, pref="equal", graphs=False):
    return {"kind": kind, "graph": "road", "rows": rows, "cols": cols, "instances": instances, "K": K,
            "wmax": wmax, "log_weights": False, "changes": changes, "mode": mode, "pref": pref,
            "canonical": False, "graphs": graphs}


def _rmat(kind, n, K, changes, mode, wmax=1000, log_weights=False, pref="equal", canonical=False,
          graphs=False):
    return {"kind": kind, "graph": "rmat", "n": n, "instances": 1, "K": K, "wmax": wmax,
            "log_weights": log_weights, "changes": changes, "mode": mode, "pref": pref,
            "canonical": canonical, "graphs": graphs}


def listed():
    cases = {
        # a site map or a test network: a few streets change, latency counts
        "update_site": _road("update", 37, 41, 2, 24, "near"),
        # a town, a few hundred streets re-weighted by the traffic
        "update_town": _road("update", 300, 311, 3, 500, "traffic"),
        # a region: streets opened and closed here and there, short detours
        "update_region": _road("update", 1000, 1000, 3, 10000, "near"),
        # the road-network benchmark's shape: long-range links appear, so that
        # nearly every path changes
        "update_road": _road("update", 1404, 1404, 3, 50000, "uniform"),
        # a small social or web graph, five objectives, odd vertex count
        "update_social": _rmat("update", 60001, 5, 3000, "uniform"),
        # the power-law benchmark's shape: distances do not fit beside the
        # parents, every parent is recovered after the update
        "update_powerlaw": _rmat("update", 1 << 22, 5, 100000, "uniform", wmax=1000000,
                                 log_weights=True, pref="ranked"),
        # many independent networks updated by one call
        "update_batched": _road("update", 140, 143, 3, 19000, "uniform", instances=64),
        # a new network is taken in: one objective's initial tree
        "scratch_road": _road("scratch", 700, 711, 1, 0, "uniform"),
        # the preferences change, the trees stay
        "combined_prefs": _road("combined", 500, 499, 6, 0, "uniform", pref="ranked"),
        # a batch is applied to a resident graph
        "apply_road": _road("apply", 1404, 1404, 3, 50000, "uniform"),
        # everything after that, on a medium power-law graph
        "step_social": _rmat("step", 1 << 18, 4, 20000, "uniform", canonical=True),
        # the whole update from pinned host buffers to host results
        "host_region": _road("host", 1000, 1000, 3, 20000, "uniform"),
    }
    return [dict(c, name=name) for name, c in cases.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["update"] * 7 + ["step", "step", "apply", "apply", "scratch", "combined", "host"])
    pref = rng.choice(["equal", "ranked"])
    graphs = kind == "update" and rng.random() < 0.25
    if rng.random() < 0.65:
        K = 1 if kind == "scratch" else rng.randint(1, 6)
        most = {"scratch": 700 * 700, "combined": 1000000, "host": 1000000}.get(kind, 5800000 // max(K, 3))
        instances = _log_int(rng, 4, 100) if kind == "update" and rng.random() < 0.25 else 1
        n = _log_int(rng, 600 * instances, most)
        cols = max(12, int(math.sqrt(n / instances) * rng.uniform(0.8, 1.25)))
        rows = max(12, n // instances // cols)
        m = 2.82 * rows * cols * instances
        changes = max(2, min(60000, int(m * math.exp(rng.uniform(math.log(2e-4), math.log(0.02))))))
        return _road(kind, rows, cols, K, changes, rng.choice(["near", "traffic", "uniform"]), instances,
                     rng.choice([10, 100, 1000]), pref, graphs)
    K = 1 if kind == "scratch" else rng.randint(1, 5)
    n = _log_int(rng, 1000, 1 << 20)
    changes = max(2, min(60000, int(16 * n * math.exp(rng.uniform(math.log(1e-4), math.log(0.01))))))
    wide = rng.random() < 0.3
    return _rmat(kind, n, K, changes, rng.choice(["traffic", "uniform"]), 1000000 if wide else 1000, wide,
                 pref, rng.random() < 0.5, graphs)


# ---------------------------------------------------------------------------
# graphs and batches, made on the GPU
# ---------------------------------------------------------------------------
def _rand_ints(gen, lo, hi, shape):
    return torch.randint(lo, hi, shape, generator=gen, device=DEV)


def _weights(case, gen, count):
    K, wmax = case["K"], case["wmax"]
    if case["log_weights"]:
        x = torch.rand((count, K), generator=gen, device=DEV)
        return torch.exp(x * math.log(wmax)).floor_().clamp_(1, wmax).to(torch.int32)
    return _rand_ints(gen, 1, wmax + 1, (count, K)).to(torch.int32)


def _road_pairs(case, gen):
    """Undirected streets of `instances` grids stored one below the other:
    70% of the grid's streets (all of the first row and column, so that the
    corner reaches the connected part) and 1% diagonals."""
    rows, cols, inst = case["rows"], case["cols"], case["instances"]
    n = rows * cols * inst
    v = torch.arange(n, device=DEV)
    x, y = v % cols, (v // cols) % rows
    keep = torch.rand((2, n), generator=gen, device=DEV) < 0.7
    right = v[(x + 1 < cols) & (keep[0] | (y == 0))]
    down = v[(y + 1 < rows) & (keep[1] | (x == 0))]
    diag = v[(x + 1 < cols) & (y + 1 < rows) & (torch.rand(n, generator=gen, device=DEV) < 0.01)]
    a = torch.cat([right, down, diag])
    b = torch.cat([right + 1, down + cols, diag + cols + 1])
    return n, a, b


def _rmat_pairs(case, gen):
    """8 n undirected R-MAT pairs (0.57, 0.19, 0.19, 0.05), ids scaled to n."""
    n = case["n"]
    levels = max(1, (n - 1).bit_length())
    count = 8 * n
    a = torch.zeros(count, dtype=torch.int64, device=DEV)
    b = torch.zeros(count, dtype=torch.int64, device=DEV)
    for _ in range(levels):
        r = torch.rand(count, generator=gen, device=DEV)
        a = 2 * a + (r >= 0.76)
        b = 2 * b + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    return n, a * n >> levels, b * n >> levels


def _graph(case, gen):
    """(n, m, row[n+1], col[m], w[m, K]) on the GPU, edge-major weights."""
    n, a, b = (_road_pairs if case["graph"] == "road" else _rmat_pairs)(case, gen)
    off = a != b
    a, b = a[off], b[off]
    keys = torch.unique(torch.cat([a * n + b, b * n + a]))
    del a, b, off
    src = torch.div(keys, n, rounding_mode="floor")
    col = (keys - src * n).to(torch.int32)
    row = torch.searchsorted(src, torch.arange(n + 1, device=DEV)).to(torch.int32)
    m = int(col.numel())
    return n, m, row, col, _weights(case, gen, m)


def _batch(case, gen, n, m, row, col):
    """Changed edges on the GPU. uniform: half random pairs, half deletions;
    near: the pairs lie at most three streets apart; traffic: existing edges
    get new weights."""
    changes = case["changes"]
    picks = _rand_ints(gen, 0, m, (changes,))
    ends = torch.searchsorted(row.to(torch.int64), picks, right=True) - 1
    edge_from, edge_to = ends.to(torch.int32), col[picks].to(torch.int32)
    if case["mode"] == "traffic":
        ins_from, ins_to = edge_from, edge_to
        del_from = del_to = torch.zeros(0, dtype=torch.int32, device=DEV)
    else:
        n_ins = (changes + 1) // 2
        part = n // case["instances"]
        u = _rand_ints(gen, 0, n, (n_ins,))
        base = torch.div(u, part, rounding_mode="floor") * part
        if case["mode"] == "near":
            cols = case["cols"]
            x = (u % cols + _rand_ints(gen, -2, 3, (n_ins,))).clamp_(0, cols - 1)
            y = (torch.div(u - base, cols, rounding_mode="floor") + _rand_ints(gen, -1, 2, (n_ins,)))
            v = base + y.clamp_(0, case["rows"] - 1) * cols + x
        else:
            v = base + _rand_ints(gen, 0, part, (n_ins,))
        v = torch.where(v == u, torch.where(u + 1 < base + part, u + 1, u - 1), v)
        ins_from, ins_to = u.to(torch.int32), v.to(torch.int32)
        del_from, del_to = edge_from[n_ins:].contiguous(), edge_to[n_ins:].contiguous()
    return {"ins_from": ins_from.contiguous(), "ins_to": ins_to.contiguous(),
            "ins_w": _weights(case, gen, int(ins_from.numel())).contiguous(),
            "del_from": del_from, "del_to": del_to}


def _capacity(case):
    """Edges that a program makes room for: the graph's, room for growth and
    the insertions of a batch."""
    if case["graph"] == "rmat":
        return 16 * case["n"] + case["changes"]
    rows, cols, inst = case["rows"], case["cols"], case["instances"]
    return 3 * rows * cols * inst + 8 * (rows + cols) * inst + 1000 + case["changes"]


def _int32(count):
    return torch.zeros(max(int(count), 1), dtype=torch.int32, device=DEV)


def _int64(count):
    return torch.zeros(max(int(count), 1), dtype=torch.int64, device=DEV)


def _tree_buffer(n, K):
    """One buffer for K trees: (buffer, distances, parents)."""
    buf = torch.zeros(12 * K * n, dtype=torch.uint8, device=DEV)
    return buf, buf[:8 * K * n].view(torch.int64), buf[8 * K * n:].view(torch.int32)


def _initial_trees(ws, n, m, row, col, columns, K, deltas, max_weights, dist, par):
    for k in range(K):
        ws.sosp_from_scratch(n, m, row, col, columns.data_ptr() + 4 * k * m, 0, deltas[k], max_weights[k],
                             dist.data_ptr() + 8 * k * n, par.data_ptr() + 4 * k * n)


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    kind, K = case["kind"], case["K"]
    n, m, row, col, w = _graph(case, gen)
    edge_w = w.reshape(-1)
    ws = mb.Workspace()
    if case["instances"] > 1:
        ws.set_sources([i * (n // case["instances"]) for i in range(case["instances"])])
    if case["canonical"]:
        ws.set_canonical_trees(True)
    if case["graphs"]:
        ws.use_graphs(True)
    pref = list(range(1, K + 1)) if case["pref"] == "ranked" else None
    deltas = [mb.default_delta(m, n, int(s)) for s in w.sum(0, dtype=torch.int64).tolist()]
    s = {"kind": kind, "ws": ws, "n": n, "m": m, "K": K, "pref": pref, "deltas": deltas,
         "max_weights": [case["wmax"]] * K}
    if kind == "apply":
        b = _batch(case, gen, n, m, row, col)
        cap = _capacity(case)
        return dict(s, row=row, col=col, w=edge_w, b=b, new_row=_int32(n + 1), new_col=_int32(cap),
                    new_w=_int32(cap * K), mask=_int32(b["ins_from"].numel()))
    columns = w.t().contiguous()
    if kind == "scratch":
        return dict(s, row=row, col=col, w=columns, dist=_int64(n), par=_int32(n))
    old, old_dist, old_par = _tree_buffer(n, K)
    _initial_trees(ws, n, m, row, col, columns, K, deltas, s["max_weights"], old_dist, old_par)
    s = dict(s, comb_dist=_int64(n), comb_par=_int32(n))
    if kind == "combined":
        return dict(s, par=old_par, keep=old)
    b = _batch(case, gen, n, m, row, col)
    if kind == "host":
        pinned = lambda t: t.cpu().pin_memory()  # noqa: E731
        out = [torch.zeros(K * n, dtype=torch.int64), torch.zeros(K * n, dtype=torch.int32),
               torch.zeros(n, dtype=torch.int64), torch.zeros(n, dtype=torch.int32),
               torch.zeros(n * K, dtype=torch.int64)]
        keep = {"graph": [pinned(t) for t in (row, col, w)], "b": {k: pinned(t) for k, t in b.items()},
                "init": [pinned(t) for t in (old_dist, old_par)], "out": [t.pin_memory() for t in out]}
        return dict(s, keep=keep, graph=[t.numpy() for t in keep["graph"]],
                    b={k: t.numpy() for k, t in keep["b"].items()},
                    init=[t.numpy() for t in keep["init"]], out=[t.numpy() for t in keep["out"]])
    # the batch applied to the resident graph, and the lists of changed edges
    n_ins, n_del = int(b["ins_from"].numel()), int(b["del_from"].numel())
    cap = _capacity(case)
    new_row, new_col, new_w = _int32(n + 1), _int32(cap), _int32(cap * K)
    mask = _int32(n_ins)
    new_m, _, _ = ws.apply_batch_device(n, K, m, row, col, edge_w, b["ins_from"], b["ins_to"], b["ins_w"],
                                        b["del_from"], b["del_to"], new_row, new_col, new_w, mask)
    lists = mb.changed_lists({"mask": mask[:n_ins].cpu().numpy().astype(np.uint32),
                              **{k: b[k].cpu().numpy() for k in ("ins_from", "ins_to", "del_from", "del_to")}}, K)
    offset = [0] + np.cumsum([len(f) for f, _ in lists]).tolist()
    both = [torch.from_numpy(np.concatenate(x + (np.zeros(1, np.int32),))).to(DEV) for x in zip(*lists)]
    trees, dist, par = _tree_buffer(n, K)
    s = dict(s, m=new_m, row=new_row, col=new_col, w=new_w, out_w=_int32(cap * K), in_row=_int32(n + 1),
             in_col=_int32(cap), in_w=_int32(cap * K), changed_from=both[0], changed_to=both[1],
             offset=offset, heads=b["ins_to"], n_heads=n_ins, old=old, trees=trees, dist=dist, par=par,
             costs=_int64(n * K) if kind == "step" else None)
    if kind == "update":
        ws.build_device_graph(n, new_m, K, new_row, new_col, new_w, s["out_w"], s["in_row"], s["in_col"],
                              s["in_w"])
    return s


def run(s):
    ws, kind, n, m, K = s["ws"], s["kind"], s["n"], s["m"], s["K"]
    if kind == "apply":
        b = s["b"]
        new_m, most, sums = ws.apply_batch_device(n, K, m, s["row"], s["col"], s["w"], b["ins_from"],
                                                  b["ins_to"], b["ins_w"], b["del_from"], b["del_to"],
                                                  s["new_row"], s["new_col"], s["new_w"], s["mask"])
        return {"m": new_m, "max": most, "sum": sums, "row": s["new_row"], "col": s["new_col"],
                "w": s["new_w"], "mask": s["mask"]}
    if kind == "scratch":
        ws.sosp_from_scratch(n, m, s["row"], s["col"], s["w"], 0, s["deltas"][0], s["max_weights"][0],
                             s["dist"], s["par"])
        return {"dist": s["dist"], "parent": s["par"]}
    if kind == "combined":
        ws.combined_sosp(n, K, s["par"], s["pref"], 0, 0, s["comb_dist"], s["comb_par"])
        return {"comb_dist": s["comb_dist"], "comb_parent": s["comb_par"]}
    if kind == "host":
        dist, par, cd, cp, costs, _ = ws.update_host(s["graph"], s["b"], s["init"][0], s["init"][1], K, 0,
                                                     pref=s["pref"], out=s["out"])
        return {"dist": dist, "parent": par, "comb_dist": cd, "comb_parent": cp, "costs": costs}
    if kind == "step":
        ws.build_device_graph(n, m, K, s["row"], s["col"], s["w"], s["out_w"], s["in_row"], s["in_col"],
                              s["in_w"])
    s["trees"].copy_(s["old"])
    ws.update_device(n, m, K, s["row"], s["col"], s["out_w"], s["in_row"], s["in_col"], s["in_w"],
                     s["changed_from"], s["changed_to"], s["offset"], s["heads"], s["n_heads"], 0,
                     s["deltas"], s["max_weights"], s["pref"], s["dist"], s["par"], s["comb_dist"],
                     s["comb_par"])
    out = {"dist": s["dist"], "parent": s["par"], "comb_dist": s["comb_dist"], "comb_parent": s["comb_par"]}
    if kind == "step":
        ws.path_costs(n, m, K, s["row"], s["col"], s["out_w"], s["comb_par"], 0, s["costs"])
        # (the order of a vertex's in-edges is not specified; the update
        # that reads them shows whether they are right)
        out.update(out_w=s["out_w"], in_row=s["in_row"], costs=s["costs"])
    return out


def work(case):
    """Every array of the pass read once (inputs) or written once (outputs)."""
    K = case["K"]
    n = case["rows"] * case["cols"] * case["instances"] if case["graph"] == "road" else case["n"]
    m = int(n * (2.82 if case["graph"] == "road" else 15.5))
    csr, graph = 4 * n + 4 * m, 4 * n + 4 * m + 4 * m * K
    trees, comb, batch = 12 * K * n, 12 * n, case["changes"] * (8 + 4 * K)
    total = {"update": 2 * graph + 2 * trees + comb + batch,
             "step": csr + 2 * 4 * m * K + graph + 2 * trees + comb + batch + 8 * K * n,
             "apply": 2 * graph + 2 * batch,
             "scratch": csr + 4 * m + 12 * n,
             "combined": 4 * K * n + comb,
             "host": graph + batch + 2 * trees + comb + 8 * K * n}[case["kind"]]
    return {"bytes": total, "flops": 0}


def exact(case, seed):
    """Every output is a whole number (ids, weights, distances, masks), so
    there is no value that rounding could move."""
    return None
