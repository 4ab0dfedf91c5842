"""Batched launch and continuous-batching server: every cost equals the
single-instance solve and the oracle, alone and in the mix; the batched
launch's whole tables equal the reference-written golden tables."""
import ctypes
import mmap
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mixed(emv):
    """80 instances of the mixed distribution (n log-uniform in [64, 4096],
    degree {3,4,6,8}, k in [4, 10], about 10% group instances)."""
    return [emv.Csr.from_stp(emv.StpInstance.mixed(777, i)) for i in range(80)]


@pytest.fixture(scope="module")
def mixed_oracle(orc, mixed):
    """The oracle's cost of every instance of `mixed`."""
    return [orc.emv_table(g.n, g.row_ptr, g.col, g.w, g.terminals, threads=16)[1] for g in mixed]


def test_batch_costs_equal_single_and_oracle(emv, mixed, mixed_oracle):
    with emv.Solver(0) as s:
        costs, stats = s.batch_solve(mixed)
        single = [s.solve(g).cost for g in mixed]
    assert list(costs) == single == mixed_oracle
    assert stats["work_items"] == len(mixed) and stats["total_ms"] > 0


def test_batch_tables_equal_reference_golden(emv, orc, golden):
    """The 24 mixed golden cases (5 of them group instances with zero-weight
    root arcs) in one batched launch: every instance's whole table hashes to
    the table the reference's own emv_kernel wrote (tests/golden/golden.json),
    and equals the oracle's cell by cell; costs equal the golden costs."""
    from tests.golden.cases import CASES, instance_for, instance_fnv

    names = sorted(n for n in CASES if n.startswith("mixed_"))
    insts = [instance_for(CASES[n]) for n in names]
    graphs = [emv.Csr.from_stp(i) for i in insts]
    with emv.Solver(0) as s:
        costs, _, tables = s.batch_solve(graphs, tables=True)
        again, _, tables2 = s.batch_solve(graphs[::-1], tables=True)  # another launch order
    groups = 0
    for name, inst, g, c, t in zip(names, insts, graphs, costs, tables):
        gold = golden["cases"][name]
        assert instance_fnv(inst) == gold["instance_fnv"]
        assert c == gold["cost"], name
        assert f"{orc.fnv64(t):016x}" == gold["table_fnv"], name
        want, _ = orc.emv_table(g.n, g.row_ptr, g.col, g.w, g.terminals, threads=8)
        assert np.array_equal(t, want), name
        groups += bool((inst.edges[:, 2] == 0).any())
    assert groups >= 3
    assert list(again[::-1]) == list(costs)
    assert all(np.array_equal(a, b) for a, b in zip(tables, tables2[::-1]))


def test_batch_merge_tile_widths_equal_reference_golden(emv, orc, golden):
    """The merge's vertex-block width (32 * mw vertices, tuned per class) and
    the relaxation's rows per chunk change only the order of the work: with
    every width forced for every class, and with the tuned tables, every
    mixed golden instance's whole table still hashes to the reference's."""
    from tests.golden.cases import CASES, instance_for

    names = sorted(n for n in CASES if n.startswith("mixed_"))
    graphs = [emv.Csr.from_stp(instance_for(CASES[n])) for n in names]
    classes = emv.BATCH_CLASSES
    with emv.Solver(0) as s:
        for mw, rcap in ((1, 32), (2, 8), (4, 128), (8, 4)):
            s.batch_set_tiles([rcap] * classes, [mw] * classes)
            costs, _, tables = s.batch_solve(graphs, tables=True)
            for name, c, t in zip(names, costs, tables):
                gold = golden["cases"][name]
                assert c == gold["cost"], (name, mw)
                assert f"{orc.fnv64(t):016x}" == gold["table_fnv"], (name, mw)
        rcap_t, mw_t = s.batch_autotune_tiles(graphs)
        costs, _, tables = s.batch_solve(graphs, tables=True)
    assert set(int(x) for x in rcap_t) <= {0, 4, 8, 16, 32, 64, 128} and rcap_t.max() > 0
    assert set(int(x) for x in mw_t) <= {0, 1, 2, 4, 8} and mw_t.max() > 0
    assert all((r > 0) == (w > 0) for r, w in zip(rcap_t, mw_t))
    for name, c, t in zip(names, costs, tables):
        assert f"{orc.fnv64(t):016x}" == golden["cases"][name]["table_fnv"], name


def test_batch_repeat_and_autotune(emv, mixed):
    with emv.Solver(0) as s:
        a, _ = s.batch_solve(mixed)
        b, _ = s.batch_solve(mixed)  # replays the captured graph
        table = s.batch_autotune(mixed)
        c, st = s.batch_solve(mixed)
    assert np.array_equal(a, b) and np.array_equal(a, c)
    assert set(int(x) for x in table) <= {0, 4, 8, 16, 32, 64, 128} and table.max() > 0


def test_batch_group_instances(emv, orc):
    groups = []
    i = 0
    while len(groups) < 6:
        inst = emv.StpInstance.mixed(4242, i)
        i += 1
        if (inst.edges[:, 2] == 0).any():
            groups.append(emv.Csr.from_stp(inst))
    with emv.Solver(0) as s:
        costs, _ = s.batch_solve(groups)
    for g, c in zip(groups, costs):
        _, want = orc.emv_table(g.n, g.row_ptr, g.col, g.w, g.terminals, threads=8)
        assert c == want


def test_batch_rejects_out_of_range(emv):
    big_k = emv.Csr.from_stp(emv.StpInstance.regular(200, 4, 1, 10, 11, 1))
    with emv.Solver(0) as s:
        with pytest.raises(emv.EmvError) as ei:
            s.batch_solve([big_k])
        assert ei.value.status == 1


@pytest.mark.parametrize("wave_sms", [0, -1, 3])
def test_server_result_same_alone_and_in_mix(emv, orc, mixed, mixed_oracle, wave_sms):
    """Continuous batching: a request's cost is the same when it runs alone
    and when it shares waves with 80 others plus a large request that runs on
    the multi-CTA path concurrently, and every served cost equals the
    oracle's (the large one's: equal to the plain GPU solve, whose table is
    pinned to the reference elsewhere).  wave_sms: the default split of the
    SMs beside a large solve, none (waves and the large solve take turns),
    and a narrow one (waves on 3 SMs, the large solve's relaxation grids on
    the rest)."""
    probe = mixed[5]
    large = emv.Csr.from_stp(emv.StpInstance.regular(70000, 8, 1, 1000, 9, 99))
    with emv.Solver(0) as s:
        want = {i: s.solve(g).cost for i, g in enumerate(mixed)}
        want_large = s.solve(large).cost
    assert [want[i] for i in range(len(mixed))] == mixed_oracle
    with emv.Server(0, hbm_budget_bytes=20 * 10**9, max_slots=256, large_n=65536, wave_sms=wave_sms) as srv:
        rid = srv.submit(probe)
        alone, _ = srv.wait(rid)
        assert alone == want[5]
        ids = {}
        lid = None
        for i, g in enumerate(mixed):
            ids[srv.submit(g)] = i
            if i == 20:
                lid = srv.submit(large)  # starts with small requests resident: the SMs are split
            if i % 10 == 0:
                time.sleep(0.002)  # arrivals while earlier requests are on the GPU
        for r, i in ids.items():
            cost, lat = srv.wait(r)
            assert cost == want[i], i
            assert lat >= 0
        assert srv.wait(lid)[0] == want_large
        st = srv.stats()
    assert st["completed"] == len(mixed) + 2
    assert st["peak_resident"] > 1 and st["waves"] >= 10


def test_server_admission_budget_and_cancel(emv, mixed):
    one = mixed[0]
    need = (one.n << one.k) * 4
    with emv.Server(0, hbm_budget_bytes=need // 2, max_slots=8) as srv:
        with pytest.raises(emv.EmvError) as ei:
            srv.submit(one)
        assert ei.value.status == 4  # EMV_ERR_OVER_BUDGET
        assert srv.stats()["rejected"] == 1
    budget = 3 * max((g.n << g.k) * 4 + 64 * g.n for g in mixed[:20])
    with emv.Server(0, hbm_budget_bytes=budget, max_slots=4) as srv:
        ids = [srv.submit(g) for g in mixed[:20]]
        srv.cancel(ids[-1])
        done = 0
        for r in ids[:-1]:
            srv.wait(r)
            done += 1
        try:
            srv.wait(ids[-1])  # finished before the cancel reached it
        except emv.EmvError as e:
            assert e.status == 10  # EMV_ERR_CANCELLED
        assert done == 19
        st = srv.stats()
    assert st["peak_resident"] <= 4 and st["peak_bytes"] <= budget


def test_autotune_first_on_fresh_context(emv):
    """Autotune samples instances by class; their cost slots are the callers'
    indices, which can exceed the sample size (a fresh context has no larger
    cost buffer from an earlier batch)."""
    graphs = [emv.Csr.from_stp(emv.StpInstance.mixed(31, i)) for i in range(300)]
    with emv.Solver(0) as s:
        table = s.batch_autotune(graphs)
        costs, _ = s.batch_solve(graphs)
        ref = [s.solve(g).cost for g in graphs[::25]]
    assert table.max() > 0
    assert list(costs[::25]) == ref


@pytest.mark.parametrize("count", [1, 2, 7, 40])
def test_batch_teams_whole_tables(emv, orc, count):
    """Few instances are solved by teams of up to 128 CTAs, many by one CTA
    each: whole tables against the oracle for a mix of sizes, an odd vertex
    count, hubs and weights past the packed arcs."""
    insts = [emv.StpInstance.regular(3001, 6, 1, 1000, 9, 1), emv.StpInstance.regular(70, 4, 1, 9, 1, 2),
             emv.StpInstance.regular(1024, 4, 1, 20000, 7, 3), emv.StpInstance.clique(150, 1, 90, 6, 4),
             emv.StpInstance.powlaw(900, 8, -0.5, 8, 1, 100, 8, 5), emv.StpInstance.regular(64, 3, 1, 9, 2, 6),
             emv.StpInstance.regular(2000, 4, 1, 100, 10, 7)]
    insts += [emv.StpInstance.mixed(99, i) for i in range(33)]
    graphs = [emv.Csr.from_stp(i) for i in insts[:count]]
    with emv.Solver(0) as s:
        costs, _, tables = s.batch_solve(graphs, tables=True)
        only, _ = s.batch_solve(graphs)
    assert np.array_equal(costs, only)
    for g, c, t in zip(graphs, costs, tables):
        want, cost = orc.emv_table(g.n, g.row_ptr, g.col, g.w, g.terminals, threads=8)
        assert np.array_equal(t, want)
        assert c == (cost if g.k > 1 else (1 << 63) - 1)


def test_batch_in_two_launches(emv):
    """A large batch is packed and launched in two parts: costs equal single
    solves in the caller's order, a faulty instance of either part is reported
    by its index (the lowest one), and the context solves again."""
    graphs = [emv.Csr.from_stp(emv.StpInstance.mixed(5, i, nmin=64, nmax=400, kmin=4, kmax=7)) for i in range(900)]
    with emv.Solver(0) as s:
        costs, st = s.batch_solve(graphs)
        again, _ = s.batch_solve(graphs)
        assert np.array_equal(costs, again) and st["work_items"] == 900
        for i in range(0, 900, 75):
            assert s.solve(graphs[i]).cost == costs[i]
        order = sorted(range(900), key=lambda i: -(graphs[i].n * 3 ** graphs[i].k))
        for faulty in ([order[0]], [order[-1]], [order[-1], order[0]], [17, 800, 400]):
            bad = list(graphs)
            for i in faulty:
                g = graphs[i]
                col = g.col.copy()
                col[3] = g.n
                bad[i] = emv.Csr(g.n, g.row_ptr, col, g.w, g.terminals)
            with pytest.raises(emv.EmvError) as ei:
                s.batch_solve(bad)
            assert ei.value.status == 1 and f"instance {min(faulty)}:" in str(ei.value)
        assert np.array_equal(s.batch_solve(graphs)[0], costs)


def test_batches_of_other_shapes_replay_the_same_graph(emv):
    """Batches whose classes, CTAs and slices differ are launched without a new
    capture (40 us of 130): taking turns costs at most a fifth more than the
    slower of them alone."""
    shapes = [[emv.Csr.from_stp(emv.StpInstance.regular(n, 4, 1, 9, 4, i)) for i in range(count)]
              for n, count in ((64, 3), (96, 4), (64, 1))]
    with emv.Solver(0) as s:
        want = [[s.solve(g).cost for g in graphs] for graphs in shapes]

        def timed(graphs):
            t0 = time.perf_counter()
            costs, _ = s.batch_solve(graphs)
            took = time.perf_counter() - t0
            assert list(costs) == want[shapes.index(graphs)]
            return took

        alone = [np.median([timed(graphs) for _ in range(40)]) for graphs in shapes]
        turns = np.median([timed(shapes[i % 3]) for i in range(120)])
    assert turns < 1.2 * max(alone)


@pytest.mark.parametrize("count,n,k", [(800, 1000, 8), (4, 20000, 10)])
def test_batch_tables_that_just_fit_the_device(emv, count, n, k):
    """A batch whose tables and graphs take nearly all free memory (all but 24 MB,
    a page of 2 MB for each of a dozen buffers) is solved, in one launch
    instead of two and without spare room, and so is the next."""
    torch = pytest.importorskip("torch")
    cudart = ctypes.CDLL("libcudart.so")
    cudart.cudaMalloc.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t]
    cudart.cudaFree.argtypes = [ctypes.c_void_p]
    one = [emv.Csr.from_stp(emv.StpInstance.regular(n, 4, 1, 9, k, seed)) for seed in range(4)]
    graphs = [one[i % 4] for i in range(count)]
    need = count * ((4 * n << k) + 4 * (n + 1) + 8 * graphs[0].arcs)
    with emv.Solver(0) as s:
        s.batch_solve([emv.Csr.from_stp(emv.StpInstance.regular(64, 4, 1, 9, 4, 1))])
        want = [s.solve(g, table=True) for g in one]
        free = torch.cuda.mem_get_info(0)[0]
        held = ctypes.c_void_p()
        assert cudart.cudaMalloc(ctypes.byref(held), free - need - (24 << 20)) == 0
        try:
            costs, _, tables = s.batch_solve(graphs, tables=True)
        finally:
            cudart.cudaFree(held)
        assert list(costs) == [want[i % 4].cost for i in range(count)]
        assert all(np.array_equal(t, want[i % 4].table) for i, t in enumerate(tables))
        assert np.array_equal(s.batch_solve(graphs)[0], costs)


def test_server_memory_follows_its_requests(emv):
    """A request whose arc slices are far larger than its table (one vertex of 62
    arcs in every slice, weights past the packed arcs) takes them once, not for
    every CTA of the GPU, and is charged for them."""
    torch = pytest.importorskip("torch")
    n, rng = 25600, np.random.default_rng(4)
    hubs = np.arange(0, n, 32)
    ends = np.stack([np.repeat(hubs, 60), rng.integers(0, n // 32, 60 * len(hubs)) * 32 + rng.integers(1, 32, 60 * len(hubs))], 1)
    ends = np.concatenate([ends, np.stack([np.arange(n - 1), np.arange(1, n)], 1)])
    edges = np.concatenate([ends, rng.integers(16384, 20000, (len(ends), 1))], 1)
    csr = emv.Csr.from_stp(emv.StpInstance(n, edges, np.array([5, 9000, 13000, 25000], np.int64)))
    assert np.diff(csr.row_ptr)[hubs].min() == 61 and np.diff(csr.row_ptr).max() <= 64
    slices = len(hubs) * 31 * 32 * 16
    with emv.Solver(0) as s:
        want = s.solve(csr).cost
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info(0)[0]
    with emv.Server(0) as srv:
        assert srv.wait(srv.submit(csr))[0] == want
        assert before - torch.cuda.mem_get_info(0)[0] < 20 * slices
        assert srv.stats()["peak_bytes"] >= slices


def test_autotune_with_a_last_slice_without_arcs(emv):
    """The autotuner takes instances unchecked: one of 1024 vertices whose last 32
    have no arcs, with more arcs than shared memory holds."""
    n, rng = 992, np.random.default_rng(6)
    ends = np.concatenate([np.stack([np.arange(n - 1), np.arange(1, n)], 1), rng.integers(0, n, (28 * n, 2))])
    ends = ends[ends[:, 0] != ends[:, 1]]
    edges = np.concatenate([ends, rng.integers(16384, 20000, (len(ends), 1))], 1)
    far = emv.Csr.from_stp(emv.StpInstance(1024, edges, np.array([5, 900], np.int64)))
    near = emv.Csr.from_stp(emv.StpInstance(n, edges, np.array([5, 900], np.int64)))
    with emv.Solver(0) as s:
        assert s.batch_autotune([far, near]).max() > 0
        assert list(s.batch_solve([near, near])[0]) == [s.solve(near).cost] * 2


def test_team_waits_for_a_long_closure(emv):
    """A team's CTAs without rows of a level wait for the one that closes its only
    row, for seconds where the closure takes a round for every vertex of a long
    band: each vertex has 64 arcs, of which the two of weight 1 are of use."""
    n = 25600
    v = np.arange(n)
    edges = np.concatenate([np.stack([v[:-j], v[j:], np.full(n - j, 1 if j == 1 else 3 * j)], 1) for j in range(1, 33)])
    csr = emv.Csr.from_stp(emv.StpInstance(n, edges, np.array([0, 5, 9, n - 1], np.int64)))
    with emv.Solver(0) as s:
        costs, st = s.batch_solve([csr])
        assert costs[0] == n - 1
        assert st["total_ms"] > 1500
        assert s.batch_solve([emv.Csr.from_stp(emv.StpInstance.regular(64, 4, 1, 9, 4, 1))])[0][0] > 0


@pytest.mark.parametrize("kind,n,degree,wmax", [("clique", 120, 0, 90), ("clique", 256, 0, 20000), ("powlaw", 400, 80, 100),
                                                ("regular", 300, 49, 30), ("regular", 1000, 180, 20000)])
def test_dense_graphs_in_one_launch_and_in_batches(emv, orc, kind, n, degree, wmax):
    """Dense graphs keep their arcs in slices up to twice the mean degree: without
    hubs, hubs only (mean degree past 254, below 5 terminals' subsets), and some
    of both."""
    if kind == "clique":
        inst = emv.StpInstance.clique(n, 1, wmax, 5, 4)
    elif kind == "powlaw":
        inst = emv.StpInstance.powlaw(n, degree, -0.5, 8, 1, wmax, 5, 4)
    else:
        inst = emv.StpInstance.regular(n, degree, 1, wmax, 5, 4)
    csr = emv.Csr.from_stp(inst)
    want, cost = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=16)
    with emv.Solver(0) as s:
        assert np.array_equal(s.solve(csr, table=True).table, want)
        assert s.solve(csr, tree=True).tree_weight == cost
        costs, _, tables = s.batch_solve([csr] * 3, tables=True)
        assert list(costs) == [cost] * 3 and all(np.array_equal(t, want) for t in tables)
        assert np.array_equal(s.sssp(csr, 7)[0], orc.sssp(csr.n, csr.row_ptr, csr.col, csr.w, 7))


@pytest.mark.parametrize("sizes,count", [((65, 70), 700), ((250, 260), 200)])
def test_dense_batches_scale_with_their_arcs(emv, sizes, count):
    """Cliques of a few per cent more vertices, across the degrees of 64 and 254,
    take at most half as long again on the device."""
    ms = []
    with emv.Solver(0) as s:
        for n in sizes:
            graphs = [emv.Csr.from_stp(emv.StpInstance.clique(n, 1, 100, 7, seed)) for seed in range(count)]
            ms.append(min(s.batch_solve(graphs)[1]["total_ms"] for _ in range(5)))
    assert ms[1] < 1.5 * ms[0]


@pytest.mark.parametrize("n", [1002, 1004])
def test_batch_tables_into_new_host_pages(emv, n):
    """Tables that go to host pages never written before take about as long as
    tables into warm buffers and a copy of their bytes into new pages together,
    whether their rows are padded on the device or not."""
    torch = pytest.importorskip("torch")
    count, size = 100, 4 * n << 8
    graphs = [emv.Csr.from_stp(emv.StpInstance.regular(n, 3, 1, 100, 8, s)) for s in range(count)]
    dev = torch.zeros((count, size // 4), dtype=torch.int32, device="cuda:0")
    costs, stats = np.zeros(count, np.int64), emv._BatchStats()

    def new_pages(bytes_):
        return np.frombuffer(mmap.mmap(-1, bytes_), np.int32)

    def timed(call):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        call()
        return time.perf_counter() - t0

    with emv.Solver(0) as s:
        insts, _keep = s._instances(graphs)

        def tables_into(bufs):
            ptrs = (ctypes.c_void_p * count)(*[b.ctypes.data for b in bufs])
            emv._check(s._lib.emv_batch_solve_tables(s._ctx, insts, count, costs.ctypes.data, ptrs, ctypes.byref(stats), None))

        warm_bufs = [new_pages(size) for _ in range(count)]
        tables_into(warm_bufs)
        warm = min(timed(lambda: tables_into(warm_bufs)) for _ in range(4))
        new, copy = [], []
        for _ in range(4):
            bufs, others = ([new_pages(size) for _ in range(count)] for _ in range(2))
            new.append(timed(lambda: tables_into(bufs)))
            copy.append(timed(lambda: [torch.from_numpy(o).copy_(d) for o, d in zip(others, dev)]))
        assert all(np.array_equal(b, w) for b, w in zip(bufs, warm_bufs))
    assert min(new) < 2 * (warm + min(copy))


@pytest.mark.parametrize("n,k", [(64, 8), (33, 10)])
def test_batches_of_a_hundred_small_dense_instances(emv, n, k):
    """Between half as many instances as CTAs and as many, teams of CTAs with less
    than a thread's work would take turns: 107 instances take at most a quarter
    longer than a CTA takes for one."""
    torch = pytest.importorskip("torch")
    ctas = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(7)
    graphs = []
    for _ in range(10):
        ends = np.concatenate([np.stack([np.arange(n - 1), np.arange(1, n)], 1), rng.integers(0, n, (16 * n, 2))])
        ends = ends[ends[:, 0] != ends[:, 1]]
        graphs.append(emv.Csr.from_stp(emv.StpInstance(n, np.concatenate([ends, rng.integers(1, 101, (len(ends), 1))], 1),
                                                       rng.choice(n, k, replace=False).astype(np.int64))))
    ms = {}
    with emv.Solver(0) as s:
        want = [s.solve(g).cost for g in graphs]
        for count in (107, 4 * ctas):  # four turns of a CTA each
            batch = [graphs[i % 10] for i in range(count)]
            for _ in range(6):
                costs, st = s.batch_solve(batch)
                ms[count] = min(ms.get(count, 1e9), st["total_ms"])
            assert list(costs) == [want[i % 10] for i in range(count)]
    assert ms[107] < 1.25 * ms[4 * ctas] / 4


def test_single_instance_batch_uses_the_gpu_as_a_solve_does(emv):
    """A batch of one gives its instance as large a team as it can use: on the
    device it takes at most a third longer than the one-launch solve."""
    n, m, k = 500, 40000, 6
    rng = np.random.default_rng(3)
    ends = np.concatenate([np.stack([np.arange(n - 1), np.arange(1, n)], 1), rng.integers(0, n, (m, 2))])
    ends = ends[ends[:, 0] != ends[:, 1]]
    g = emv.Csr.from_stp(emv.StpInstance(n, np.concatenate([ends, rng.integers(1, 101, (len(ends), 1))], 1),
                                         rng.choice(n, k, replace=False).astype(np.int64)))
    with emv.Solver(0) as s:
        solves, batches = [], []
        for _ in range(8):
            r = s.solve(g)
            assert r.timing["relax_launches"] == 1
            solves.append(r.timing["kernel_ms"])
            costs, st = s.batch_solve([g])
            assert costs[0] == r.cost
            batches.append(st["total_ms"])
    assert min(batches) < 1.33 * min(solves)
