"""GPU parity: the sm_103a solver against the oracle and the reference's golden tables.

The bar is bit-exact: the whole int32 DP table and the cost equal the
oracle's on the same instance and the reference's golden hashes; the tree is a
valid Steiner tree of real edges whose weight equals the cost.
"""
import ctypes
import os
import subprocess
import time

import numpy as np
import pytest

from tests.golden.cases import CASES, instance_for, instance_fnv
from tests.helpers import check_tree, table_row_fnv

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def solver(emv):
    s = emv.Solver(0)
    yield s
    s.close()


@pytest.mark.parametrize("name", sorted(CASES))
def test_table_and_cost_match_oracle_and_golden(name, emv, orc, golden, solver):
    g = golden["cases"][name]
    inst = instance_for(CASES[name])
    assert instance_fnv(inst) == g["instance_fnv"]
    csr = emv.Csr.from_stp(inst)
    res = solver.solve(csr, tree=True, table=True)
    want, want_cost = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=8)
    assert res.cost == want_cost == g["cost"]
    mism = np.argwhere(res.table != want)
    assert mism.size == 0, f"{len(mism)} cells differ, first (X, v) = {mism[:5].tolist()}"
    assert f"{orc.fnv64(res.table):016x}" == g["table_fnv"]
    if "row_fnv" in g and csr.k <= 8:
        assert table_row_fnv(res.table) == g["row_fnv"]
    check_tree(csr.n, inst.edges, res.tree, csr.terminals, res.cost)
    assert res.tree_weight == res.cost or csr.k == 1


def test_repeat_solves_identical(emv, solver):
    inst = emv.StpInstance.regular(5000, 6, 1, 1000, 9, 77)
    csr = emv.Csr.from_stp(inst)
    a = solver.solve(csr, table=True)
    b = solver.solve(csr, table=True)
    assert a.cost == b.cost and np.array_equal(a.table, b.table)


def test_kernel_dev_on_caller_table(emv, orc, solver):
    torch = pytest.importorskip("torch")
    inst = emv.StpInstance.regular(3000, 8, 1, 1000, 7, 31337)
    csr = emv.Csr.from_stp(inst)
    dev = torch.device("cuda:0")
    row = torch.from_numpy(csr.row_ptr).to(dev)
    col = torch.from_numpy(csr.col).to(dev)
    w = torch.from_numpy(csr.w).to(dev)
    ld = csr.n + 5  # any stride >= n
    table = torch.full(((1 << csr.k), ld), -7, dtype=torch.int32, device=dev)
    stream = torch.cuda.current_stream().cuda_stream
    cost = solver.kernel_dev(csr.n, csr.arcs, row.data_ptr(), col.data_ptr(), w.data_ptr(), csr.terminals,
                             table.data_ptr(), ld, stream)
    torch.cuda.synchronize()
    want, want_cost = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=8)
    got = table[:, :csr.n].cpu().numpy()
    assert cost == want_cost
    assert np.array_equal(got, want)
    assert (table[:, csr.n:].cpu().numpy() == -7).all(), "padding columns must stay untouched"


def test_solve_dev_matches_solve(emv, solver):
    torch = pytest.importorskip("torch")
    inst = emv.StpInstance.regular(2500, 4, 1, 100, 8, 5)
    csr = emv.Csr.from_stp(inst)
    dev = torch.device("cuda:0")
    row, col, w = (torch.from_numpy(a).to(dev) for a in (csr.row_ptr, csr.col, csr.w))
    torch.cuda.synchronize()
    r1 = solver.solve_dev(csr.n, csr.arcs, row.data_ptr(), col.data_ptr(), w.data_ptr(), csr.terminals, tree=True)
    r2 = solver.solve(csr)
    assert r1.cost == r2.cost
    check_tree(csr.n, inst.edges, r1.tree, csr.terminals, r1.cost)


def test_sssp_matches_oracle(emv, orc, solver):
    inst = emv.StpInstance.regular(20000, 6, 1, 1000, 2, 8)
    csr = emv.Csr.from_stp(inst)
    for s in (0, 12345, 19999):
        d, _ = solver.sssp(csr, s)
        assert np.array_equal(d, orc.sssp(csr.n, csr.row_ptr, csr.col, csr.w, s))


def test_large_single_solve_properties(emv, orc, solver):
    """n = 1e5, degree 20, k = 12 (the single large solve): the full table is
    too slow for the oracle here, so check it through size-independent
    properties plus exact rows over the first 5 terminals (d[X][v] depends on
    the terminals of X only; the oracle computes those 32 rows)."""
    inst = emv.StpInstance.regular(100000, 20, 1, 100, 12, 123456789)
    csr = emv.Csr.from_stp(inst)
    res = solver.solve(csr, tree=True, table=True)
    t = res.table
    sub, _ = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals[:5], threads=16)
    assert np.array_equal(t[:32], sub)
    assert (t[0] == emv.INF32).all() and (t[1:] < emv.INF32).all()
    rng = np.random.default_rng(0)
    src = np.repeat(np.arange(csr.n), np.diff(csr.row_ptr))
    for X in rng.integers(1, 1 << 12, size=24):
        row = t[X]
        # closure: d[X][v] <= d[X][u] + w(u, v) for every arc
        assert (row[csr.col] <= row[src] + csr.w).all()
        # monotone in X and bounded by every split
        for b in range(12):
            if X >> b & 1:
                assert (t[X ^ (1 << b)] <= row).all()
                Y = X & ~(1 << b)
                if Y:
                    assert (row <= t[Y] + t[1 << b]).all()
    assert res.cost == int(t[(1 << 11) - 1, csr.terminals[11]])
    check_tree(csr.n, inst.edges, res.tree, csr.terminals, res.cost)


@pytest.mark.parametrize("n,degree,k", [(700, 6, 13), (300, 4, 14), (120, 4, 15)])
def test_large_k_whole_table(emv, orc, solver, n, degree, k):
    """k = 13..15 run the streamed merge in subset groups with row tiles; the
    whole table must still equal the oracle's."""
    inst = emv.StpInstance.regular(n, degree, 1, 1000, k, 4242 + k)
    csr = emv.Csr.from_stp(inst)
    res = solver.solve(csr, tree=True, table=True)
    want, want_cost = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=8)
    assert res.cost == want_cost
    mism = np.argwhere(res.table != want)
    assert mism.size == 0, f"{len(mism)} cells differ, first (X, v) = {mism[:5].tolist()}"
    check_tree(csr.n, inst.edges, res.tree, csr.terminals, res.cost)


def _narrow_levels(table, terms):
    """Levels the solver takes with 16-bit values, recomputed from the
    oracle's table: M(j) is the largest value level j's merge writes (from the
    lower levels, terminal override included), M(1) the largest single-source
    distance.  Level m >= 2 relaxes with 16-bit records when M(m-1) + M(1) <=
    32767; level m >= 3 merges from 16-bit rows when every M(j) + M(m-j) <=
    65533.  Returns (relaxed, merged) level counts."""
    k = len(terms)
    M = {1: int(max(table[1 << i].max() for i in range(k)))}
    for m in range(2, k):
        mx = 0
        for X in range(1, 1 << k):
            if bin(X).count("1") != m:
                continue
            best = None
            Y = (X - 1) & X
            while Y:
                if Y < (X ^ Y):
                    s = table[Y].astype(np.int64) + table[X ^ Y]
                    best = s if best is None else np.minimum(best, s)
                Y = (Y - 1) & X
            for t in range(k):
                if X >> t & 1:
                    best[terms[t]] = table[X ^ (1 << t)][terms[t]]
            mx = max(mx, int(best.max()))
        M[m] = mx
    relaxed = sum(1 for m in range(2, k + 1) if M[m - 1] + M[1] <= 32767)
    merged = sum(1 for m in range(3, k + 1) if max(M[j] + M[m - j] for j in range(1, m // 2 + 1)) <= 65533)
    return relaxed, merged


# weight range -> which levels take 16-bit relaxation records and merge rows
WIDTH_CASES = {100: ("all", "all"), 3000: ("some", "all"), 5000: ("some", "some"), 8000: ("none", "none")}


@pytest.mark.parametrize("ew", sorted(WIDTH_CASES))
def test_value_widths_match_oracle(emv, orc, ew):
    """16-bit values are taken per level only where the level maxima bound
    them: weights up to 100 keep every level 16-bit, larger weights the lower
    levels only or none.  The level counts equal the rule's, and the table
    equals the oracle's with automatic and with 32-bit values."""
    k = 10
    inst = emv.StpInstance.regular(6000, 6, 1, ew, k, 515)
    csr = emv.Csr.from_stp(inst)
    want, want_cost = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=8)
    relaxed, merged = _narrow_levels(want, list(csr.terminals))
    kinds = tuple("all" if c == top else "none" if c == 0 else "some" for c, top in ((relaxed, k - 1), (merged, k - 2)))
    assert kinds == WIDTH_CASES[ew]
    with emv.Solver(0) as s:
        for bits in (0, 32):
            s.set_value_bits(bits)
            res = s.solve(csr, tree=True, table=True)
            assert res.timing["relax16_levels"] == (relaxed if bits == 0 else 0)
            assert res.timing["merge16_levels"] == (merged if bits == 0 else 0)
            assert res.cost == want_cost
            mism = np.argwhere(res.table != want)
            assert mism.size == 0, f"bits {bits}: {len(mism)} cells differ, first (X, v) = {mism[:5].tolist()}"
            check_tree(csr.n, inst.edges, res.tree, csr.terminals, res.cost)
        with pytest.raises(emv.EmvError):
            s.set_value_bits(16)


def test_wide_records_and_partial_merge_block_equal_32_bit_values(emv):
    """Records past three quarters of L2 (n = 2^18 + 40) take 1 KB per vertex:
    512 rows of 16 bits against 256 of 32; the last 64-vertex merge block is
    partial.  Both tables are identical."""
    inst = emv.StpInstance.regular((1 << 18) + 40, 6, 1, 100, 11, 2718)
    csr = emv.Csr.from_stp(inst)
    with emv.Solver(0) as s:
        a = s.solve(csr, table=True)
        s.set_value_bits(32)
        b = s.solve(csr, table=True)
    assert a.timing["relax16_levels"] == 10 and a.timing["merge16_levels"] == 9
    assert b.timing["relax16_levels"] == 0 and b.timing["merge16_levels"] == 0
    assert a.cost == b.cost and np.array_equal(a.table, b.table)


def test_640_byte_records_match_oracle(emv, orc):
    """k = 12 with weights up to 8000 keeps 32-bit values: levels 5..7 (792,
    924, 792 subsets) relax in 5, 6 and 5 chunks of 640-byte records instead
    of 7, 8 and 7 of 512 bytes.  Whole table against the oracle, and the
    launch count of that chunk rule."""
    inst = emv.StpInstance.regular(2000, 6, 1, 8000, 12, 606)
    csr = emv.Csr.from_stp(inst)
    want, want_cost = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=8)
    with emv.Solver(0) as s:
        res = s.solve(csr, tree=True, table=True)
    assert res.timing["relax16_levels"] == 0
    # level 1, then per level m: 66 -> 1, 220 -> 2, 495 -> 4, 792 -> 5, 924 -> 6, 792 -> 5, 495 -> 4, 220 -> 2,
    # 66, 12, 1 -> 1 each
    assert res.timing["relax_launches"] == 1 + 1 + 2 + 4 + 5 + 6 + 5 + 4 + 2 + 1 + 1 + 1
    assert res.cost == want_cost
    mism = np.argwhere(res.table != want)
    assert mism.size == 0, f"{len(mism)} cells differ, first (X, v) = {mism[:5].tolist()}"
    check_tree(csr.n, inst.edges, res.tree, csr.terminals, res.cost)


def test_bad_inputs_report_status(emv, solver):
    disc = emv.StpInstance.from_text(
        "section graph\nnodes 4\nedges 2\ne 1 2 3\ne 3 4 5\nend\nsection terminals\nterminals 2\nt 1\nt 3\nend\n")
    csr = emv.Csr.from_stp(disc)
    with pytest.raises(emv.EmvError) as ei:
        solver.solve(csr)
    assert ei.value.status == 7  # EMV_ERR_DISCONNECTED
    inst = emv.StpInstance.regular(100, 4, 1, 10, 5, 1)
    csr = emv.Csr.from_stp(inst)
    with pytest.raises(emv.EmvError) as ei:
        solver.solve(csr, terminals=[0, 1, 200])
    assert ei.value.status == 1
    with pytest.raises(emv.EmvError):
        solver.solve(csr, terminals=list(range(21)))
    # the context stays usable after errors
    assert solver.solve(csr).cost > 0


def test_admission_checks_on_every_entry_point(emv, solver):
    """Weights near 2^30 are EMV_ERR_OVERFLOW, a head out of range
    EMV_ERR_BAD_INPUT and a disconnected graph EMV_ERR_DISCONNECTED, from the
    host entry point with its default flags and from both device entry
    points (the device check of k_pack_scan and the level-1 connectivity
    test), and from emv_closure_noalloc; the context solves again after each."""
    torch = pytest.importorskip("torch")
    dev = torch.device("cuda:0")
    stream = torch.cuda.current_stream().cuda_stream
    base = emv.Csr.from_stp(emv.StpInstance.regular(300, 4, 1, 100, 5, 21))
    heavy = emv.Csr(base.n, base.row_ptr, base.col, np.full_like(base.w, 1 << 28), base.terminals)
    bad_head = emv.Csr(base.n, base.row_ptr, base.col.copy(), base.w, base.terminals)
    bad_head.col[11] = base.n + 5
    disc_inst = emv.StpInstance(8, np.array([[0, 1, 3], [1, 2, 4], [3, 4, 1], [4, 5, 2], [6, 7, 1], [5, 6, 9]],
                                            np.int64), np.array([0, 2, 4], np.int64))
    disc = emv.Csr.from_stp(disc_inst)
    disc = emv.Csr(disc.n, disc.row_ptr, disc.col, disc.w, disc.terminals)
    # vertices 0-2 and 3-7 are two components
    assert disc.n == 8
    cases = [(heavy, 8), (bad_head, 1), (disc, 7)]
    for g, status in cases:
        with pytest.raises(emv.EmvError) as ei:
            solver.solve(g)
        assert ei.value.status == status
        row, col, w = (torch.from_numpy(a).to(dev) for a in (g.row_ptr, g.col, g.w))
        with pytest.raises(emv.EmvError) as ei:
            solver.solve_dev(g.n, g.arcs, row.data_ptr(), col.data_ptr(), w.data_ptr(), g.terminals, stream=stream)
        assert ei.value.status == status
        table = torch.empty(((1 << g.k), g.n), dtype=torch.int32, device=dev)
        with pytest.raises(emv.EmvError) as ei:
            solver.kernel_dev(g.n, g.arcs, row.data_ptr(), col.data_ptr(), w.data_ptr(), g.terminals,
                              table.data_ptr(), g.n, stream)
        assert ei.value.status == status
        torch.cuda.synchronize()
    # the closure entry point: a single weight of 2^30 or more, and a head out of range
    huge = emv.Csr(base.n, base.row_ptr, base.col, base.w.copy(), base.terminals)
    huge.w[3] = 1 << 30
    init = torch.full((1, base.n), emv.INF32, dtype=torch.int32, device=dev)
    init[0, 0] = 0
    for g, status in ((huge, 8), (bad_head, 1)):
        row, col, w = (torch.from_numpy(a).to(dev) for a in (g.row_ptr, g.col, g.w))
        with pytest.raises(emv.EmvError) as ei:
            emv.Solver.closure_noalloc(g.n, g.arcs, row.data_ptr(), col.data_ptr(), w.data_ptr(), init.data_ptr(), 1,
                                       g.n, init.data_ptr(), stream)
        assert ei.value.status == status
    # still usable
    assert solver.solve(base).cost == solver.solve(base, check=False).cost > 0


def test_sweep_limit_is_a_timeout_status_and_context_survives(emv, orc):
    """A bounded device loop that runs out reports EMV_ERR_TIMEOUT through the
    status word; nothing traps and the same context solves again."""
    inst = emv.StpInstance.regular(3000, 4, 1, 1000, 6, 99)
    csr = emv.Csr.from_stp(inst)
    want = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals)[1]
    with emv.Solver(0) as s:
        s.set_sweep_limit(2)
        with pytest.raises(emv.EmvError) as ei:
            s.solve(csr)
        assert ei.value.status == 5  # EMV_ERR_TIMEOUT
        s.set_sweep_limit(0)
        assert s.solve(csr).cost == want
        with pytest.raises(emv.EmvError):
            s.set_sweep_limit(-1)


def test_table_beyond_device_memory_is_oom_and_context_survives(emv, solver):
    """A table larger than the device (n * 2^k * 4 bytes well above its memory)
    fails its allocation with EMV_ERR_OOM; the context is usable afterwards."""
    torch = pytest.importorskip("torch")
    total = torch.cuda.get_device_properties(0).total_memory
    k = 20
    n = 1 << 14
    while n * (4 << k) < 2 * total:
        n <<= 1
    inst = emv.StpInstance.regular(n, 4, 1, 10, k, 5)
    csr = emv.Csr.from_stp(inst)
    with pytest.raises(emv.EmvError) as ei:
        solver.solve(csr)
    assert ei.value.status == 3  # EMV_ERR_OOM
    small = emv.Csr.from_stp(emv.StpInstance.regular(500, 4, 1, 10, 5, 5))
    assert solver.solve(small).cost > 0


def test_cli_reference_lines(emv, tmp_path):
    """reader-el-gpu -el -list prints the reference's lines; the regexes are
    those of the reference's scripts (experiments/verify.py:126-147)."""
    import re

    inst = emv.StpInstance.regular(3000, 4, 1, 1000, 9, 2718)
    csr = emv.Csr.from_stp(inst)
    cost = emv.Solver().solve(csr).cost
    inst.cost = cost
    path = str(tmp_path / "i.stp")
    inst.write(path)
    out = subprocess.run([emv.CLI_PATH, "-in", path, "-el", "-list"], stdout=subprocess.PIPE, text=True,
                         check=True).stdout
    line = next(ln for ln in out.splitlines() if ln.startswith("erickson"))
    mt = re.search(r"erickson: \[zero:(.*)ms\] \[kernel:(.*)ms (.*)GiB/s\] \[traceback: (.*)ms\] done. "
                   r"\[(.*)ms\] \[cost:(.*)] {peak:(.*)GiB} {curr:(.*)GiB}", line)
    assert mt and int(mt.group(6)) == cost
    inp = next(ln for ln in out.splitlines() if ln.startswith("input"))
    assert re.search(r"(.*)n = (.*), m = (.*), k = (.*), cost = (.*) \[(.*)ms\] {peak:(.*)GiB} {curr:(.*)GiB}", inp)
    sol = next(ln for ln in out.splitlines() if ln.startswith("solution"))
    pairs = re.findall(r'"([^"]*)"', sol)
    lookup = {}
    for u, v, w in inst.edges:
        lookup.setdefault((min(u, v), max(u, v)), set()).add(int(w))
    tree = []
    for p in pairs:
        u, v = (int(x) - 1 for x in p.split())
        tree.append((u, v, min(lookup[(min(u, v), max(u, v))])))
    check_tree(inst.n, inst.edges, np.array(tree), inst.terminals, cost)
    # a wrong cost line in the input ends the run with ERROR, as in the reference
    inst.cost = cost + 1
    inst.write(path)
    r = subprocess.run([emv.CLI_PATH, "-in", path, "-el"], stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True)
    assert r.returncode != 0 and "min_cost != cost" in r.stderr


def test_cli_dijkstra_command(emv, orc, tmp_path):
    """-dijkstra (R:2454-2484): source = rand() % n after srand(seed), distances on the GPU."""
    import ctypes
    import re

    inst = emv.StpInstance.regular(5000, 6, 1, 1000, 3, 4)
    path = str(tmp_path / "d.stp")
    inst.write(path)
    out = subprocess.run([emv.CLI_PATH, "-in", path, "-dijkstra", "-seed", "77"], stdout=subprocess.PIPE, text=True,
                         check=True).stdout
    mt = re.search(r"dijkstra: \[source: (\d+)\] \[total: (.*) ms (.*)GiB/s\] \[reached: (\d+)\] \[max: (\d+)\]", out)
    assert mt, out
    libc = ctypes.CDLL(None)
    libc.srand(77)
    src = libc.rand() % inst.n
    assert int(mt.group(1)) == src + 1
    csr = emv.Csr.from_stp(inst)
    d = orc.sssp(csr.n, csr.row_ptr, csr.col, csr.w, src)
    assert int(mt.group(4)) == inst.n and int(mt.group(5)) == int(d.max())


def test_roofline_scale_solve(emv, orc, tmp_path):
    """n = 2^20, degree 10, k = 14 (the 64 GiB table).  With the fixture of
    tests/golden/make_roofline_golden.py (the reference's own complete run on
    the host cores): the whole table hashes to the reference's table and the
    costs are equal.  Without it: d[X][v] depends only on the terminals in X,
    so the reference's run on the first 10 terminals (ref_emv -kprefix 10:
    the 1024 rows X < 2^10) pins those rows bit for bit (the oracle's first 6
    terminals where the reference leg is not built).  Closure and
    monotonicity on sampled rows either way."""
    import json

    torch = pytest.importorskip("torch")
    from tests.golden.make_roofline_golden import OUT as GOLDEN, SPEC, instance_fnv_fast

    inst = emv.StpInstance.regular(SPEC["n"], SPEC["degree"], SPEC["wmin"], SPEC["wmax"], SPEC["k"], SPEC["seed"])
    csr = emv.Csr.from_stp(inst)
    dev = torch.device("cuda:0")
    row, col, w = (torch.from_numpy(a).to(dev) for a in (csr.row_ptr, csr.col, csr.w))
    n, k = csr.n, csr.k
    table = torch.empty(((1 << k), n), dtype=torch.int32, device=dev)
    with emv.Solver(0) as s:
        cost = s.kernel_dev(n, csr.arcs, row.data_ptr(), col.data_ptr(), w.data_ptr(), csr.terminals,
                            table.data_ptr(), n, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert cost == int(table[(1 << (k - 1)) - 1, int(csr.terminals[k - 1])])

    def rows_fnv(x0, x1, h=orc.FNV_BASIS, per_row=False):
        rows = []
        for X0 in range(x0, x1, 256):
            part = table[X0:min(x1, X0 + 256)].cpu().numpy()
            h = orc.fnv64(part, h)
            if per_row:
                rows += [orc.fnv64(part[i]) for i in range(part.shape[0])]
        return h, rows

    if os.path.exists(GOLDEN):
        with open(GOLDEN) as f:
            gold = json.load(f)
        assert instance_fnv_fast(orc, inst) == gold["instance_fnv"]
        assert cost == gold["cost"]
        h, _ = rows_fnv(0, 1 << k)
        assert f"{h:016x}" == gold["table_fnv"], "whole table differs from the reference's"
    elif orc.reference_available():
        kp = 10
        path = str(tmp_path / "roofline.stp")
        inst.write(path)
        rowfnv = str(tmp_path / "rows.bin")
        r = orc.ref_emv(path, kprefix=kp, rowfnv_out=rowfnv, threads=os.cpu_count())
        ref_rows = np.fromfile(rowfnv, dtype="<u8")
        assert r["k"] == kp and ref_rows.size == 1 << kp
        h, got_rows = rows_fnv(0, 1 << kp, per_row=True)
        bad = np.nonzero(np.array(got_rows, dtype=np.uint64) != ref_rows)[0]
        assert bad.size == 0, f"{bad.size} rows differ from the reference, first subsets {bad[:8].tolist()}"
        assert h == r["fnv"]
        # the cost of the 10-terminal prefix instance is a cell of the full table
        assert r["cost"] == int(table[(1 << (kp - 1)) - 1, int(csr.terminals[kp - 1])])
    else:
        want, _ = orc.emv_table(n, csr.row_ptr, csr.col, csr.w, csr.terminals[:6], threads=16)
        assert np.array_equal(table[:64].cpu().numpy(), want)
    src = np.repeat(np.arange(n), np.diff(csr.row_ptr))
    rng = np.random.default_rng(3)
    for X in rng.integers(1 << 10, 1 << k, size=4):
        r = table[int(X)].cpu().numpy()
        assert (r[csr.col] <= r[src] + csr.w).all()
        for b in range(k):
            if X >> b & 1 and X ^ (1 << b):
                assert (table[int(X) ^ (1 << b)].cpu().numpy() <= r).all()
    del table
    torch.cuda.empty_cache()


@pytest.mark.parametrize("n,degree,k,dup", [(64, 3, 1, False), (64, 3, 2, False), (300, 4, 3, False),
                                            (301, 4, 6, True), (5000, 6, 9, False)])
def test_calls_without_a_table_equal_whole_table_solves(emv, orc, solver, n, degree, k, dup):
    """A call that returns no table computes the rows over the first k - 1
    terminals only: its cost and tree are those of the whole-table solve,
    also with a repeated terminal and for k = 1 and 2."""
    inst = emv.StpInstance.regular(n, degree, 1, 50, k, 31 + k)
    csr = emv.Csr.from_stp(inst)
    terms = csr.terminals.copy()
    if dup:
        terms[-1] = terms[1]
    csr = emv.Csr(csr.n, csr.row_ptr, csr.col, csr.w, terms)
    _, want = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=8)
    whole = solver.solve(csr, tree=True, table=True)
    for res in (solver.solve(csr, tree=True), solver.solve(csr, tree=True, all_rows=True)):
        assert res.cost == whole.cost == want
        assert np.array_equal(res.tree, whole.tree) and res.tree_weight == whole.tree_weight
    if k <= 10:
        costs, _ = solver.batch_solve([csr])
        assert int(costs[0]) == want


ONE_LAUNCH = {  # graph, k: the one-launch solver's edges
    "one_slice": (("regular", 32, 3, 1, 9), 5),
    "odd_n_many_rows": (("regular", 65, 4, 1, 50), 11),
    "registers_two_pairs": (("regular", 1024, 4, 1, 1000), 6),
    "pairs_past_the_registers": (("regular", 999, 10, 1, 100), 5),
    "arcs_in_shared_memory": (("regular", 4096, 10, 1, 1024), 4),
    "arcs_in_global_memory": (("regular", 12002, 8, 1, 100), 4),
    "largest_weight_packed": (("regular", 1500, 4, 16383, 16383), 4),
    "smallest_weight_not_packed": (("regular", 1500, 4, 16383, 16384), 4),
    "hubs_only": (("clique", 200, 0, 1, 20000), 5),
    "hubs_and_leaves": (("powlaw", 5000, 8, 1, 100), 6),
    "most_vertices": (("regular", 29000, 4, 1, 30), 3),
}


@pytest.mark.parametrize("name", sorted(ONE_LAUNCH))
def test_one_launch_solver_whole_table(emv, orc, solver, name):
    """Small instances run as one launch: whole table against the oracle, from
    host memory and into a caller's table of an odd stride."""
    torch = pytest.importorskip("torch")
    (kind, n, degree, wmin, wmax), k = ONE_LAUNCH[name]
    if kind == "clique":
        inst = emv.StpInstance.clique(n, wmin, wmax, k, 17)
    elif kind == "powlaw":
        inst = emv.StpInstance.powlaw(n, degree, -0.5, 8, wmin, wmax, k, 17)
    else:
        inst = emv.StpInstance.regular(n, degree, wmin, wmax, k, 17)
    csr = emv.Csr.from_stp(inst)
    want, want_cost = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=8)
    res = solver.solve(csr, tree=True, table=True)
    assert res.timing["relax_launches"] == 1
    assert res.cost == want_cost and np.array_equal(res.table, want)
    check_tree(csr.n, inst.edges, res.tree, csr.terminals, res.cost)
    row, col, w = (torch.from_numpy(a).to("cuda:0") for a in (csr.row_ptr, csr.col, csr.w))
    ld = csr.n + 3 - csr.n % 2
    table = torch.full(((1 << k), ld), -7, dtype=torch.int32, device="cuda:0")
    cost = solver.kernel_dev(csr.n, csr.arcs, row.data_ptr(), col.data_ptr(), w.data_ptr(), csr.terminals,
                             table.data_ptr(), ld, torch.cuda.current_stream().cuda_stream)
    got = table.cpu().numpy()
    assert cost == want_cost and np.array_equal(got[:, :csr.n], want) and (got[:, csr.n:] == -7).all()


@pytest.mark.parametrize("kind,n,degree,wmax", [("regular", 2, 1, 9), ("regular", 8192, 4, 1000), ("regular", 8193, 6, 100),
                                                ("powlaw", 40000, 8, 100), ("regular", 100000, 20, 100)])
def test_sssp_sizes_match_oracle(emv, orc, solver, kind, n, degree, wmax):
    """Distances of one source on both sides of the one-launch solver's limit
    and with hubs, a disconnected vertex included (INT64_MAX)."""
    make = emv.StpInstance.powlaw if kind == "powlaw" else emv.StpInstance.regular
    inst = make(n, degree, -0.5, 8, 1, wmax, 2, 8) if kind == "powlaw" else make(n + n * degree % 2, degree, 1, wmax, 2, 8)
    alone = emv.StpInstance(inst.n + 1, inst.edges, inst.terminals)
    for g in (emv.Csr.from_stp(inst), emv.Csr.from_stp(alone)):
        for s in (0, g.n - 1):
            d, _ = solver.sssp(g, s)
            assert np.array_equal(d, orc.sssp(g.n, g.row_ptr, g.col, g.w, s))


@pytest.mark.parametrize("k", [3, 6, 12])
def test_level1_record_widths(emv, orc, solver, k):
    """Level-1 records of 4, 8 and 16 rows in front of the record kernels
    (a graph past the one-launch solver)."""
    inst = emv.StpInstance.regular(33000, 4, 1, 1000, k, 77)
    csr = emv.Csr.from_stp(inst)
    res = solver.solve(csr, table=True)
    for i, t in enumerate(csr.terminals):
        d = orc.sssp(csr.n, csr.row_ptr, csr.col, csr.w, int(t))
        assert np.array_equal(res.table[1 << i], d)


@pytest.mark.parametrize("n,k,wmax,bits", [(33000, 5, 100, 0), (33000, 7, 100, 0), (33000, 9, 5000, 0), (33000, 8, 100, 32),
                                           (6000, 10, 8000, 0)])
def test_hubs_in_the_record_kernels(emv, orc, n, k, wmax, bits):
    """Power-law graphs past the one-launch solver: vertices of up to a thousand
    arcs are relaxed by whole blocks, in every record width and both value
    widths.  Whole table against the oracle."""
    inst = emv.StpInstance.powlaw(n, 8, -0.5, 8, 1, wmax, k, 5)
    csr = emv.Csr.from_stp(inst)
    assert np.diff(csr.row_ptr).max() > 256
    want, cost = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=16)
    with emv.Solver(0) as s:
        s.set_value_bits(bits)
        for check in (True, False):
            res = s.solve(csr, table=True, check=check)
            assert res.cost == cost and np.array_equal(res.table, want)


@pytest.mark.parametrize("n,wmin,wmax,k", [(64, 1, 9, 2), (500, 0, 1, 9), (2000, 0, 2, 12), (40000, 0, 3, 6)])
def test_traceback_pieces_and_zero_weight_runs(emv, orc, solver, n, wmin, wmax, k):
    """The pieces of a tree are walked by different warps; runs of zero-weight
    arcs share one set of search arrays between them.  Valid trees of the
    optimal weight, the same on every call."""
    csr = emv.Csr.from_stp(inst := emv.StpInstance.regular(n, 4, wmin, wmax, k, 3))
    first = solver.solve(csr, tree=True)
    check_tree(csr.n, inst.edges, first.tree, csr.terminals, first.cost)
    again = solver.solve(csr, tree=True, all_rows=True)
    assert again.cost == first.cost and again.tree_weight == first.tree_weight


def test_traceback_of_a_long_path(emv, solver):
    """More edges than come back with the first copy."""
    n = 5000
    edges = np.stack([np.arange(n - 1), np.arange(1, n), np.ones(n - 1, np.int64)], axis=1).astype(np.int64)
    inst = emv.StpInstance(n, edges, np.array([0, 2500, n - 1], np.int64))
    res = solver.solve(emv.Csr.from_stp(inst), tree=True)
    assert res.cost == n - 1
    check_tree(n, edges, res.tree, inst.terminals, res.cost)


RECORD_CLOSURES = {
    # kind: n, degree, wmin, wmax, k, value bits
    "one warp": (33, 4, 1, 9, 12, 0),
    "zero weights": (64, 4, 0, 0, 12, 0),
    "long arcs": (6001, 20, 1, 100, 12, 0),
    "short arcs": (5000, 21, 90, 100, 12, 0),
    "long arcs 32 bits": (6001, 20, 1, 100, 12, 32),
    "values above 16 bits": (3000, 10, 1, 100000, 12, 0),
    "several windows a warp": (200002, 3, 1, 1000, 4, 0),
}


@pytest.mark.parametrize("kind", sorted(RECORD_CLOSURES))
def test_arcs_ruled_out_by_the_excesses(emv, orc, kind):
    """Record closures skip arcs that no row of a record can use: whole table
    against the oracle where few and where most arcs are skipped."""
    n, degree, wmin, wmax, k, bits = RECORD_CLOSURES[kind]
    csr = emv.Csr.from_stp(emv.StpInstance.regular(n, degree, wmin, wmax, k, 11))
    want, cost = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=16)
    with emv.Solver(0) as s:
        s.set_value_bits(bits)
        res = s.solve(csr, table=True)
        assert res.timing["relax_launches"] > 1
        assert res.cost == cost and np.array_equal(res.table, want)


@pytest.mark.parametrize("k", [3, 12])
def test_record_closures_with_unreached_and_isolated_vertices(emv, orc, solver, k):
    """Weights above 32768 beside 16-bit distances, a component without a
    terminal and vertices without arcs: values of a row may be unreached."""
    rng = np.random.default_rng(3)
    n = 20040
    a = emv.StpInstance.regular(20000, 4, 1, 40, k, 2)
    heavy = np.stack([rng.integers(0, 10000, 3000), rng.integers(10000, 20000, 3000), rng.integers(30000, 70000, 3000)], axis=1)
    far = np.stack([np.arange(20000, 20029), np.arange(20001, 20030), np.full(29, 7)], axis=1)
    for edges, lost in ((np.concatenate([a.edges, heavy]), 0), (np.concatenate([a.edges, heavy, far]), 40)):
        inst = emv.StpInstance(n if lost else 20000, edges.astype(np.int64), a.terminals)
        csr = emv.Csr.from_stp(inst)
        want, cost = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=16)
        res = solver.solve(csr, table=True, check=not lost)
        assert res.cost == cost and np.array_equal(res.table, want)


@pytest.mark.parametrize("n,degree,wmax,k,bits", [(9001, 5, 50, 12, 0), (20011, 6, 10000, 7, 0), (20011, 20, 100, 9, 32),
                                                  (160001, 4, 1000, 5, 0)])
def test_levels_of_few_rows_on_narrow_records(emv, orc, n, degree, wmax, k, bits):
    """Levels of 1 to 36 rows: merged rows closed on narrow records of every
    width, beside wider levels that read their 16-bit copies."""
    csr = emv.Csr.from_stp(emv.StpInstance.regular(n + n * degree % 2, degree, 1, wmax, k, 4))
    want, cost = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=16)
    with emv.Solver(0) as s:
        s.set_value_bits(bits)
        res = s.solve(csr, table=True)
        assert res.cost == cost and np.array_equal(res.table, want)


@pytest.mark.parametrize("n,degree,k", [(5001, 8, 10), (9000, 6, 11), (16384, 3, 10), (16385, 4, 10), (15002, 20, 9),
                                        (14998, 20, 7)])
def test_one_launch_limits_on_caller_tables(emv, orc, solver, n, degree, k):
    """Both sides of the one-launch solver's limits on vertices and arcs from 10
    terminals on: whole caller table and the cost-only solve."""
    torch = pytest.importorskip("torch")
    csr = emv.Csr.from_stp(emv.StpInstance.regular(n + n * degree % 2, degree, 1, 200, k, 23))
    want, want_cost = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=16)
    row, col, w = (torch.from_numpy(a).to("cuda:0") for a in (csr.row_ptr, csr.col, csr.w))
    ld = csr.n + 3 - csr.n % 2
    table = torch.full(((1 << k), ld), -7, dtype=torch.int32, device="cuda:0")
    cost = solver.kernel_dev(csr.n, csr.arcs, row.data_ptr(), col.data_ptr(), w.data_ptr(), csr.terminals,
                             table.data_ptr(), ld, torch.cuda.current_stream().cuda_stream)
    got = table.cpu().numpy()
    assert cost == want_cost and np.array_equal(got[:, :csr.n], want) and (got[:, csr.n:] == -7).all()
    assert solver.solve(csr, tree=True).cost == want_cost


def test_traceback_waits_for_long_zero_weight_searches(emv, solver):
    """All weights 0: every piece of the tree is one search over a large part of
    the graph, and the pieces queue for the search's arrays for seconds."""
    csr = emv.Csr.from_stp(inst := emv.StpInstance.regular(1 << 19, 4, 0, 0, 12, 3))
    solver.solve(csr)
    t0 = time.perf_counter()
    res = solver.solve(csr, tree=True)
    took = 1e3 * (time.perf_counter() - t0)
    assert res.cost == 0 and res.tree_weight == 0
    check_tree(csr.n, inst.edges, res.tree, csr.terminals, 0)
    assert 0.9 * took < res.timing["kernel_ms"] + res.timing["traceback_ms"] < took


def test_refused_one_launch_solve_traces_nothing(emv, solver):
    """A small graph whose value bound reaches 2^30 is refused without a walk
    through the table: with a tree requested the refusal takes no longer than
    half of the walk through the rows that the solve before it left there."""
    n = 20000
    edges = np.stack([np.arange(n - 1), np.arange(1, n), np.ones(n - 1, np.int64)], axis=1).astype(np.int64)
    good = emv.Csr.from_stp(emv.StpInstance(n, edges, np.array([0, n - 1, n - 2], np.int64)))
    far = edges.copy()
    far[[5, 6], 2] = 2**30 - 1
    bad = emv.Csr.from_stp(emv.StpInstance(n, far, good.terminals.astype(np.int64)))
    walk = solver.solve(good, tree=True).timing["traceback_ms"]
    assert walk > 4.0
    for _ in range(3):
        solver.solve(good)
        t0 = time.perf_counter()
        with pytest.raises(emv.EmvError) as ei:
            solver.solve(bad, tree=True)
        took = 1e3 * (time.perf_counter() - t0)
        assert ei.value.status == 8
        assert took < walk / 2


@pytest.mark.parametrize("n", [300, 40000])
def test_refused_graphs_leave_the_callers_table_alone(emv, solver, n):
    """emv_kernel_dev on a graph that its check refuses writes no cell."""
    torch = pytest.importorskip("torch")
    g = emv.Csr.from_stp(emv.StpInstance.regular(n, 4, 1, 9, 4, 5))
    table = torch.full((1 << 4, n), -7, dtype=torch.int32, device="cuda:0")
    for array, value, status in (("col", n, 1), ("w", -1, 1), ("w", 2**30 - 1, 8)):
        arrays = {name: getattr(g, name).copy() for name in ("row_ptr", "col", "w")}
        arrays[array][10:14] = value
        row, col, w = (torch.from_numpy(arrays[x]).to("cuda:0") for x in ("row_ptr", "col", "w"))
        with pytest.raises(emv.EmvError) as ei:
            solver.kernel_dev(n, g.arcs, row.data_ptr(), col.data_ptr(), w.data_ptr(), g.terminals, table.data_ptr(), n,
                              torch.cuda.current_stream().cuda_stream)
        assert ei.value.status == status
        assert bool((table == -7).all())


def test_out_of_memory_for_the_tree_leaves_no_work_behind(emv):
    """A one-launch solve that cannot have the traceback's buffers fails before
    it enqueues anything: the caller may free its arrays on return."""
    torch = pytest.importorskip("torch")
    cudart = ctypes.CDLL("libcudart.so")
    cudart.cudaMalloc.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t]
    cudart.cudaFree.argtypes = [ctypes.c_void_p]
    g = emv.Csr.from_stp(emv.StpInstance.regular(24000, 4, 1, 9, 10, 5))
    stream = torch.cuda.Stream()
    held = []
    with emv.Solver(0) as s:
        want = s.solve(g, stream=stream.cuda_stream).cost
        size = 1 << 36
        while size >= 1 << 16:
            p = ctypes.c_void_p()
            if cudart.cudaMalloc(ctypes.byref(p), size) == 0:
                held.append(p)
            else:
                cudart.cudaGetLastError()
                size >>= 1
        try:
            with pytest.raises(emv.EmvError) as ei:
                s.solve(g, tree=True, stream=stream.cuda_stream)
            idle = stream.query()
        finally:
            for p in held:
                cudart.cudaFree(p)
        assert ei.value.status == 3 and idle
        assert s.solve(g, tree=True, stream=stream.cuda_stream).cost == want


@pytest.mark.parametrize("side,limit", [(100, 110), (200, 210), (316, 340)])
def test_sweep_limit_holds_for_long_frontiers(emv, side, limit):
    """Grids need about a sweep of the record kernels for a row of vertices;
    closures that move a change by one arc a sweep take twice as many within
    the same cap."""
    at = np.arange(side * side).reshape(side, side)
    ends = np.concatenate([np.stack([at[:, :-1].ravel(), at[:, 1:].ravel()], 1),
                           np.stack([at[:-1].ravel(), at[1:].ravel()], 1)])
    w = np.random.default_rng(side + 77).integers(1, 101 if side > 300 else 11, len(ends))
    terms = np.random.default_rng(1).choice(side * side, size=5, replace=False)
    csr = emv.Csr.from_stp(emv.StpInstance(side * side, np.concatenate([ends, w[:, None]], 1), terms.astype(np.int64)))
    with emv.Solver(0) as s:
        want, dist = s.solve(csr).cost, s.sssp(csr, 1)[0]
        s.set_sweep_limit(limit)
        assert s.solve(csr).cost == want
        assert np.array_equal(s.sssp(csr, 1)[0], dist)
        s.set_sweep_limit(limit // 8)
        with pytest.raises(emv.EmvError) as ei:
            s.solve(csr)
        assert ei.value.status == 5


def test_sssp_of_many_arcs_takes_the_whole_gpu(emv, orc, solver):
    """One CTA does not read all arcs of a dense graph: its kernel takes no more
    than twice the time of the same graph with leaves past the one-launch limit."""
    n, m = 8192, 500000
    rng = np.random.default_rng(n)
    ends = rng.integers(0, n, (m, 2))
    ends = np.concatenate([ends[ends[:, 0] != ends[:, 1]], np.stack([np.arange(n - 1), np.arange(1, n)], 1)])
    leaves = np.arange(n, 8200)
    more = np.concatenate([ends, np.stack([leaves % n, leaves], 1)])
    ms = []
    for count, e in ((n, ends), (8200, more)):
        w = rng.integers(1, 51, len(e))
        g = emv.Csr.from_stp(emv.StpInstance(count, np.concatenate([e, w[:, None]], 1), np.array([0], np.int64)))
        assert np.array_equal(solver.sssp(g, 1)[0], orc.sssp(g.n, g.row_ptr, g.col, g.w, 1))
        ms.append(min(solver.sssp(g, 1)[1] for _ in range(5)))
    assert ms[0] < 2 * ms[1]


@pytest.mark.parametrize("n,degree,k,wmax,one", [(20011, 8, 9, 100, True), (24000, 12, 5, 100, False), (30000, 4, 4, 100, True),
                                                 (30000, 8, 4, 100, False), (20000, 14, 8, 30000, False),
                                                 (4000, 20, 11, 100, True), (4000, 60, 12, 100, False),
                                                 (16000, 8, 12, 100, False), (12000, 17, 11, 100, False)])
def test_one_launch_for_as_many_arcs_as_it_reads_faster(emv, orc, solver, n, degree, k, wmax, one):
    """Both sides of the line on vertices, arcs and terminals up to which a
    small solve runs in one launch."""
    csr = emv.Csr.from_stp(emv.StpInstance.regular(n + n * degree % 2, degree, 1, wmax, k, 29))
    want, cost = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=16)
    for table in (False, True):
        res = solver.solve(csr, table=table)
        assert res.cost == cost and (res.timing["relax_launches"] == 1) == one
    assert np.array_equal(res.table, want)


@pytest.mark.parametrize("hubs", [1, 10, 100])
def test_sssp_of_crowded_arcs_stays_in_one_launch(emv, orc, solver, hubs):
    """Half of the arcs at a few neighbouring vertices: the closure takes no longer
    than 0.4 ms (a warp of the narrow records 0.5 to 1.6)."""
    n, m = 5368, 91000
    rng = np.random.default_rng(hubs)
    ends = np.concatenate([np.stack([rng.integers(0, hubs, m), rng.integers(0, n, m)], 1),
                           np.stack([np.arange(n - 1), np.arange(1, n)], 1)])
    ends = ends[ends[:, 0] != ends[:, 1]]
    g = emv.Csr.from_stp(emv.StpInstance(n, np.concatenate([ends, rng.integers(1, 1001, (len(ends), 1))], 1), np.array([0], np.int64)))
    assert np.array_equal(solver.sssp(g, n // 2)[0], orc.sssp(g.n, g.row_ptr, g.col, g.w, n // 2))
    assert min(solver.sssp(g, n // 2)[1] for _ in range(5)) < 0.4


@pytest.mark.parametrize("check", [True, False])
def test_crowded_graphs_past_the_line_run_in_one_launch(emv, orc, solver, check):
    """Half of the arcs at a hundred vertices: past the line on arcs and vertices
    such a graph still runs as one launch, from host and from device memory, and
    the same size without hubs does not."""
    torch = pytest.importorskip("torch")
    n, m, k = 14000, 135000, 3
    rng = np.random.default_rng(6)
    path = np.stack([np.arange(n - 1), np.arange(1, n)], 1)
    for hubs in (100, n):
        ends = np.concatenate([path, np.stack([rng.integers(0, hubs, m), rng.integers(0, n, m)], 1)])
        ends = ends[ends[:, 0] != ends[:, 1]]
        g = emv.Csr.from_stp(emv.StpInstance(n, np.concatenate([ends, rng.integers(1, 101, (len(ends), 1))], 1),
                                             rng.choice(n, k, replace=False).astype(np.int64)))
        want, cost = orc.emv_table(g.n, g.row_ptr, g.col, g.w, g.terminals, threads=16)
        res = solver.solve(g, table=True, tree=True, check=check)
        assert res.cost == cost == res.tree_weight and np.array_equal(res.table, want)
        assert (res.timing["relax_launches"] == 1) == (hubs == 100)
        row, col, w = (torch.from_numpy(a).to("cuda:0") for a in (g.row_ptr, g.col, g.w))
        table = torch.empty((1 << k, n), dtype=torch.int32, device="cuda:0")
        assert solver.kernel_dev(n, g.arcs, row.data_ptr(), col.data_ptr(), w.data_ptr(), g.terminals, table.data_ptr(), n,
                                 torch.cuda.current_stream().cuda_stream) == cost
        assert np.array_equal(table.cpu().numpy(), want)
