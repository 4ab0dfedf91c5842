"""What is measured of the solver: the calls its users make, over their range.

A case is one kind of call on one kind of instance:

  host     ``Solver.solve`` on a host CSR with the tree (and, for small
           instances, the table): what the command line and scripts call
  device   ``Solver.kernel_dev`` on a device CSR and a caller-owned device
           table, whose whole contents are the output
  batch    ``Solver.batch_solve`` on many mixed instances after the autotuner
  serve    a burst of requests through ``Server``, 2 % of them large
  sssp     ``Solver.sssp``, the single-source distances of one vertex
  closure  ``Solver.closure_noalloc``, the closure of up to 32 device rows

Every output is a whole number (costs, distances, table cells, tree edges).
"""
from __future__ import annotations

import numpy as np
import torch

import steiner_edge_linear_gb300 as E

INT64_MAX = (1 << 63) - 1
LARGE = dict(n=1 << 17, degree=8, wmin=1, wmax=1000, k=12)  # the serving stream's large requests

# A program keeps one solver and one server per process, whatever it solves.
_kept: dict = {}


def _solver() -> E.Solver:
    if "solver" not in _kept:
        _kept["solver"] = E.Solver(0)
    return _kept["solver"]


def _server() -> E.Server:
    if "server" not in _kept:
        _kept["server"] = E.Server(0)
    return _kept["server"]


def listed() -> list[dict]:
    return [
        # the smallest instances of a test set (SteinLib-sized), with the tree: launches and latency
        dict(name="host n64 k4", call="host", graph="regular", n=64, degree=3, wmax=10, k=4, table=False),
        # the plain instance of the benchmark configurations: cost, tree and the whole table
        dict(name="host n1024 k8", call="host", graph="regular", n=1024, degree=4, wmax=1000, k=8, table=True),
        # an ordinary instance solved one at a time, with the tree
        dict(name="host n4096 k10", call="host", graph="regular", n=4096, degree=10, wmax=1024, k=10, table=False),
        # a middle-sized graph with an odd vertex count and stride, few terminals
        dict(name="device n20011 k9", call="device", graph="regular", n=20011, degree=8, wmax=1000, k=9),
        # the single large plain solve of the benchmark configurations
        dict(name="device n100000 k12", call="device", graph="regular", n=100000, degree=20, wmax=100, k=12),
        # the serving stream's large request, solved alone from host memory, with the tree
        dict(name="host n2^17 k12", call="host", graph="regular", n=1 << 17, degree=8, wmax=1000, k=12, table=False),
        # a graph whose working set exceeds L2 (the roofline-scale graph with fewer terminals)
        dict(name="device n2^20 k10", call="device", graph="regular", n=1 << 20, degree=10, wmax=1024, k=10),
        # power-law degrees (hubs of a thousand arcs) and weights that need 32-bit values
        dict(name="device powlaw n30000 k10", call="device", graph="powlaw", n=30000, degree=10, wmax=8000, k=10),
        # the batched configuration: 4096 mixed instances in one launch
        dict(name="batch 4096", call="batch", count=4096),
        # a burst of the serving stream: mixed requests and 2 % large ones
        dict(name="serve 400", call="serve", count=392, large=8),
        # the -dijkstra command's call
        dict(name="sssp n100000", call="sssp", graph="regular", n=100000, degree=20, wmax=100, k=2),
        # the allocation-free closure close to its limits, odd sizes
        dict(name="closure n131071 r31", call="closure", graph="regular", n=131071, degree=8, wmax=1000, k=2, rows=31),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng) -> dict:
    call = rng.choices(["host", "device", "batch", "serve", "sssp", "closure"], [30, 30, 13, 5, 11, 11])[0]
    if call == "batch":
        return dict(call=call, count=_log_int(rng, 24, 4096))
    if call == "serve":
        return dict(call=call, count=_log_int(rng, 40, 392), large=rng.randint(0, 6))
    top = {"host": 1 << 17, "device": 1 << 20, "sssp": 1 << 20, "closure": 131072}[call]
    graph = rng.choices(["regular", "powlaw", "clique"], [75, 15, 10])[0]
    if graph == "clique":
        n, degree = _log_int(rng, 40, 1500), 0
        arcs = n * (n - 1)
    else:
        n = _log_int(rng, 512 if graph == "powlaw" else 64, top)
        degree = rng.choice([6, 8, 10] if graph == "powlaw" else [3, 4, 6, 8, 10, 20])
        n += n * degree % 2
        n = min(n, top)
        arcs = n * degree
    # the solver takes graphs whose summed edge weights stay below 2^30
    wmax = min(rng.choice([10, 100, 1000, 1024, 8000]), max(1, int(1.5 * 2**31 / arcs)))
    case = dict(call=call, graph=graph, n=n, degree=degree, wmax=wmax, k=2)
    if call == "closure":
        case["rows"] = rng.randint(1, 32)
    if call in ("host", "device"):
        k = rng.randint(3, 12)
        while k > 3 and (n * 3**k > 6e10 or n << k > 1 << 30):
            k -= 1
        case["k"] = k
    if call == "host":
        case["table"] = n << case["k"] <= 1 << 20
    return case


def _csr(case: dict, seed: int) -> E.Csr:
    if case["graph"] == "powlaw":
        inst = E.StpInstance.powlaw(case["n"], case["degree"], -0.5, 8, 1, case["wmax"], case["k"], seed)
    elif case["graph"] == "clique":
        inst = E.StpInstance.clique(case["n"], 1, case["wmax"], case["k"], seed)
    else:
        inst = E.StpInstance.regular(case["n"], case["degree"], 1, case["wmax"], case["k"], seed)
    return E.Csr.from_stp(inst)


def _mixed(count: int, seed: int) -> list[E.Csr]:
    return [E.Csr.from_stp(E.StpInstance.mixed(seed * 8192, i)) for i in range(count)]


def _large(index: int, seed: int) -> E.Csr:
    return E.Csr.from_stp(E.StpInstance.regular(seed=seed * 8192 + index, **LARGE))


def _stream_order(case: dict, small: list, large: list) -> list:
    """The large requests spread evenly among the small ones."""
    if not large:
        return small
    out, step = [], max(1, len(small) // len(large))
    for i, g in enumerate(small):
        if i % step == 0 and i // step < len(large):
            out.append(large[i // step])
        out.append(g)
    return out + large[-(-len(small) // step):]


def prepare(case: dict, seed: int) -> dict:
    call = case["call"]
    state = {"call": call}
    if call == "batch":
        state["solver"] = _solver()
        state["graphs"] = _mixed(case["count"], seed)
        if "tuned" not in _kept:  # once per program, on instances of the kind it will solve
            _kept["tuned"] = state["solver"].batch_autotune_tiles(_mixed(1024, 77))
        return state
    if call == "serve":
        state["server"] = _server()
        state["graphs"] = _stream_order(case, _mixed(case["count"], seed),
                                        [_large(i, seed) for i in range(case["large"])])
        return state
    g = _csr(case, seed)
    if call in ("host", "sssp"):
        state.update(solver=_solver(), graph=g, table=case.get("table", False), source=seed % g.n)
        return state
    dev = torch.device("cuda", 0)
    state.update(solver=_solver(), n=g.n, arcs=g.arcs, terms=g.terminals,
                 csr=[torch.from_numpy(a).to(dev) for a in (g.row_ptr, g.col, g.w)])
    if call == "device":
        state["out"] = torch.zeros((1 << case["k"], g.n), dtype=torch.int32, device=dev)
    else:
        state["init"] = _init_rows(case, seed).to(dev)
        state["out"] = torch.zeros_like(state["init"])
    return state


def _init_rows(case: dict, seed: int) -> torch.Tensor:
    """Rows to close: a few seeded vertices each (as merged rows seed a relaxation), the rest INF."""
    gen = torch.Generator().manual_seed(seed)
    n, rows = case["n"], case["rows"]
    init = torch.full((rows, n), E.INF32, dtype=torch.int32)
    for r in range(rows):
        at = torch.randint(0, n, (1 + r % 5,), generator=gen)
        init[r, at] = torch.randint(0, 2 * case["wmax"], (at.numel(),), generator=gen, dtype=torch.int32)
    return init


def run(state: dict):
    call = state["call"]
    if call == "host":
        r = state["solver"].solve(state["graph"], tree=True, table=state["table"])
        tree = np.zeros((state["graph"].n, 3), np.int32)  # the edges, then zeros: as many rows for every instance
        tree[:r.tree.shape[0]] = r.tree
        out = {"cost": r.cost, "tree": tree, "tree_weight": r.tree_weight}
        if state["table"]:
            out["table"] = r.table
        return out
    if call == "batch":
        return state["solver"].batch_solve(state["graphs"])[0]
    if call == "serve":
        srv = state["server"]
        return np.array([srv.wait(i)[0] for i in [srv.submit(g) for g in state["graphs"]]], np.int64)
    if call == "sssp":
        return state["solver"].sssp(state["graph"], state["source"])[0]
    row, col, w = (t.data_ptr() for t in state["csr"])
    out, stream = state["out"], torch.cuda.current_stream().cuda_stream
    if call == "device":
        cost = state["solver"].kernel_dev(state["n"], state["arcs"], row, col, w, state["terms"], out.data_ptr(),
                                          out.stride(0), stream)
        return {"cost": cost, "table": out}
    E.Solver.closure_noalloc(state["n"], state["arcs"], row, col, w, state["init"].data_ptr(), out.shape[0],
                             state["n"], out.data_ptr(), stream)
    return out


def _arcs(case: dict) -> int:
    return case["n"] * (case["n"] - 1 if case["graph"] == "clique" else case["degree"])


def _solve_work(n: int, arcs: int, k: int, table: bool) -> tuple[float, float]:
    """(bytes, operations): the graph once and, where it is an output, the
    table once; an add and a minimum per unordered subset pair and vertex, and
    per row and arc.  A call that returns no table needs the rows of the
    subsets of the first k - 1 terminals only: the cost is the cell of those
    k - 1 terminals at the last one, and every row depends only on the rows of
    its own subsets."""
    if not table:
        k = max(1, k - 1)
    rows = (1 << k) - 1
    pairs = (3**k - 2 ** (k + 1) + 1) / 2
    return 4.0 * (n + 1) + 8.0 * arcs + 4.0 * n * (rows + 1) * table, 2.0 * n * pairs + 2.0 * rows * arcs


def work(case: dict) -> dict:
    call = case["call"]
    if call in ("batch", "serve"):
        sizes = [(g.n, g.arcs, g.k) for g in _mixed(case["count"], 1)]
        sizes += [(LARGE["n"], LARGE["n"] * LARGE["degree"], LARGE["k"])] * case.get("large", 0)
        parts = [_solve_work(*s, False) for s in sizes]
        return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}
    n, arcs = case["n"], _arcs(case)
    if call == "sssp":
        return {"bytes": 4.0 * (n + 1) + 8.0 * arcs + 8.0 * n, "flops": 2.0 * arcs}
    if call == "closure":
        return {"bytes": 4.0 * (n + 1) + 8.0 * arcs + 8.0 * n * case["rows"], "flops": 2.0 * arcs * case["rows"]}
    b, f = _solve_work(n, arcs, case["k"], case.get("table", call == "device"))
    return {"bytes": b, "flops": f}


# ------------------------------------------------- the same outputs in plain 64-bit torch

class _Closure:
    """min-plus closure of int64 rows by Bellman-Ford rounds over the arcs."""

    def __init__(self, g: E.Csr):
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        deg = torch.from_numpy(np.diff(g.row_ptr).astype(np.int64))
        self.tail = torch.repeat_interleave(torch.arange(g.n), deg).to(dev)
        self.head = torch.from_numpy(g.col.astype(np.int64)).to(dev)
        self.w = torch.from_numpy(g.w.astype(np.int64)).to(dev)
        self.dev = dev

    def __call__(self, rows: torch.Tensor) -> torch.Tensor:
        while True:
            cand = torch.clamp(rows[:, self.head] + self.w, max=E.INF32)
            new = rows.scatter_reduce(1, self.tail.expand(rows.shape[0], -1), cand, "amin")
            if torch.equal(new, rows):
                return rows
            rows = new


def _table64(g: E.Csr) -> torch.Tensor:
    close, k = _Closure(g), g.k
    terms = [int(t) for t in g.terminals]
    t = torch.full((1 << k, g.n), E.INF32, dtype=torch.int64, device=close.dev)
    for m in range(1, k + 1):
        level = [x for x in range(1, 1 << k) if bin(x).count("1") == m]
        rows = torch.full((len(level), g.n), E.INF32, dtype=torch.int64, device=close.dev)
        for i, x in enumerate(level):
            if m == 1:
                rows[i, terms[x.bit_length() - 1]] = 0
                continue
            y = (x - 1) & x
            while 2 * y > x or y > x ^ y:
                rows[i] = torch.minimum(rows[i], t[y] + t[x ^ y])
                y = (y - 1) & x
            for b in range(k):
                if x >> b & 1:
                    rows[i, terms[b]] = t[x ^ (1 << b), terms[b]]
        t[level] = close(rows)
    return t


def exact(case: dict, seed: int):
    call = case["call"]
    if call in ("batch", "serve"):
        return None
    g = _csr(case, seed)
    if call == "sssp":
        close = _Closure(g)
        row = torch.full((1, g.n), E.INF32, dtype=torch.int64, device=close.dev)
        row[0, seed % g.n] = 0
        d = close(row)[0]
        return torch.where(d >= E.INF32, INT64_MAX, d).cpu().numpy()
    if call == "closure":
        close = _Closure(g)
        return close(_init_rows(case, seed).to(torch.int64).to(close.dev)).to(torch.int32)
    if 3**g.k > 100_000 or g.arcs << g.k > 1 << 29:
        return None
    t = _table64(g)
    cost = int(t[(1 << (g.k - 1)) - 1, int(g.terminals[g.k - 1])])
    if call == "host":
        out = {"cost": cost, "tree": None, "tree_weight": cost}
        if case["table"]:
            out["table"] = t.to(torch.int32).cpu().numpy()
        return out
    return {"cost": cost, "table": t.to(torch.int32)}
