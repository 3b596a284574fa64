"""Device scan and sort through the entry points that rest on them, at the
sizes where a tile, a block or a look-back step begins or ends."""
import numpy as np
import pytest

from misfit_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb():
    from misfit_gb300 import native
    native.load_library()
    return native


# one block holds 1,024 items; 256-item tiles up to 192 of them (32 per look-back step), then 2,048-item tiles
SCAN_SIZES = [1, 31, 32, 33, 1023, 1024, 1025, 1280, 1281, 33 * 256, 33 * 256 + 1, 49151, 49152, 49153, 51200, 51201,
              33 * 2048 + 7, 300001]


@pytest.mark.parametrize("lines", SCAN_SIZES)
def test_line_scan_at_tile_edges(gb, lines, tmp_path):
    """Every kept line lands at the exclusive count of the kept lines before it."""
    rng = np.random.default_rng(lines)
    n = 1000
    u = rng.integers(1, n + 1, size=lines)
    v = rng.integers(1, n + 1, size=lines)
    comment = rng.random(lines) < 0.3
    path = str(tmp_path / "1.mtx")
    with open(path, "w") as f:
        f.write("".join("%% %d\n" % a if c else "%d %d\n" % (a, b) for a, b, c in zip(u, v, comment)))
    keep = ~comment & (u != v)
    with gb.Graph.from_csr(*W.er_graph(n, 4, 1)) as g:
        gu, gv, ins = g.parse_batch_file(path)
        assert np.array_equal(ins, g.flag_updates(gu, gv))
    assert np.array_equal(gu, u[keep] - 1) and np.array_equal(gv, v[keep] - 1)


# one block sorts 256 / 1,024 / 2,048 / 4,096 / 8,192 pairs, longer inputs take 2,048-pair tiles; a batch of m lines
# sorts m pairs, its 2m endpoint slots and its appended entries
@pytest.mark.parametrize("m", [1, 2, 128, 129, 256, 257, 512, 513, 1024, 1025, 2048, 2049, 4096, 4097, 8192, 8193, 16385])
def test_batch_sorts_at_block_edges(gb, m):
    """Pairs repeated within the batch (grouping in batch order), vertices repeated (previous occurrence, order of
    appended entries), free flags: rows, degrees, membership and cluster ids equal the oracle's."""
    import oracle as O
    n = 3000
    nindex, nlist = W.er_graph(n, 6, 2)
    mis = O.greedy_mis(nindex, nlist)
    orc = O.Oracle.from_csr(nindex, nlist)
    rng = np.random.default_rng(m)
    with gb.Graph.from_csr(nindex, nlist) as g:
        g.set_mis(mis)
        orc.set_mis(mis)
        for _ in range(2):
            u = rng.integers(0, n, m)
            hot = rng.random(m) < 0.3
            u[hot] = rng.integers(0, 3, hot.sum())
            v = (u + 1 + rng.integers(0, np.where(hot, 40, n - 1))) % n
            flip = rng.random(m) < 0.5
            u, v = np.where(flip, v, u).astype(np.int32), np.where(flip, u, v).astype(np.int32)
            ins = rng.integers(0, 2, m).astype(np.uint8)
            orc.apply_batch(u, v, ins)
            g.apply_batch(u, v, ins)
            assert np.array_equal(g.degrees(), orc.degrees())
            for x in np.unique(np.concatenate([u, v]))[:300]:
                assert np.array_equal(g.row(int(x)), orc.row(int(x))), x
            assert np.array_equal(g.get_mis(), orc.get_mis())
            assert np.array_equal(g.cluster_ids(), orc.cluster_ids())


# one block plans up to 4,096 lines; the first 160 sub-batches come back with the plan, the rest by a copy
@pytest.mark.parametrize("m,max_csr", [(700, 100000), (1500, 40000), (4096, 200000), (4097, 200000), (5000, 60000)])
def test_plan_cuts(gb, m, max_csr):
    """Many short sub-batches (and re-plans after the limit grows): cuts, limit, membership and ids equal the oracle's."""
    import oracle as O
    n = 2500
    nindex, nlist = W.er_graph(n, 5, 7)
    mis = O.greedy_mis(nindex, nlist)
    orc = O.Oracle.from_csr(nindex, nlist)
    u, v, ins = W.ToggleStream(n, nindex, nlist, m).next_batch(m, with_flags=True)
    with gb.Graph.from_csr(nindex, nlist) as g:
        for x in (g, orc):
            x.max_csr = max_csr
            x.set_mis(mis)
        g.trace(True)
        orc.trace(True)
        g.apply_batch(u, v, ins)
        orc.apply_batch(u, v, ins)
        a, b = g.trace_records(), orc.trace_records()
        assert len(a) == len(b)
        for x, y in zip(a, b):
            assert np.array_equal(x[0][[0, 1, 2, 3, 5, 6, 7]], np.asarray(y[0])[[0, 1, 2, 3, 5, 6, 7]])
        assert g.max_csr == orc.max_csr
        assert np.array_equal(g.get_mis(), orc.get_mis())
        assert np.array_equal(g.cluster_ids(), orc.cluster_ids())


@pytest.mark.parametrize("hub,push", [(120, 0), (126, 0), (127, 1), (128, 0), (129, 1), (140, 2)])
def test_row_length_limit_of_short_kernels(gb, hub, push):
    """Graphs of rows up to 128 positions take the group-per-row kernels, longer ones the general path: a hub row
    that starts at `hub` entries and grows by a few every batch crosses the line; every stage equals the oracle's."""
    import oracle as O
    n = 1500
    rng = np.random.default_rng(hub)
    nindex, nlist = W.er_graph(n, 5, hub)
    lo, hi = W.undirected_pairs(n, nindex, nlist)
    keep = (lo != 7) & (hi != 7)
    others = rng.permutation(np.delete(np.arange(n), 7))
    nindex, nlist = W.csr_from_pairs(n, np.concatenate([lo[keep], np.full(hub, 7)]),
                                     np.concatenate([hi[keep], others[:hub]]))
    mis = O.greedy_mis(nindex, nlist)
    orc = O.Oracle.from_csr(nindex, nlist)
    stream = W.ToggleStream(n, nindex, nlist, hub)
    with gb.Graph.from_csr(nindex, nlist) as g:
        g.set_tuning(cand_push=push)
        for x in (g, orc):
            x.set_mis(mis)
            x.trace(True)
        for b in range(4):
            u, v, ins = stream.next_batch(150, with_flags=True)
            more = others[hub + 2 * b:hub + 2 * b + 2].astype(np.int32)
            u, v = np.concatenate([u, more]), np.concatenate([v, np.full(2, 7, np.int32)])
            ins = np.concatenate([ins, np.ones(2, np.uint8)])
            g.apply_batch(u, v, ins)
            orc.apply_batch(u, v, ins)
            a, b2 = g.trace_records(), orc.trace_records()
            assert len(a) == len(b2)
            for x, y in zip(a, b2):
                for field in (1, 2, 3, 4, 5):
                    assert np.array_equal(x[field], y[field]), field
            assert np.array_equal(g.get_mis(), orc.get_mis())


# one block commits up to 1,024 edges, another up to 16,384 edges with up to 8,192 writes; more go to host-driven rounds
@pytest.mark.parametrize("m,writes", [(1000, 900), (1024, 1024), (1025, 1025), (1100, 600), (8300, 8192), (8300, 8193),
                                      (16384, 5000), (16385, 5000), (9000, 9000)])
def test_repair_commit_blocks(gb, m, writes):
    """One sub-batch of m edges, `writes` of them inserts that join two members (each removes one), the rest inserts
    around them: dependent chains, joins and plain removals; order, membership and ids equal the oracle's."""
    import oracle as O
    n = 45000
    rng = np.random.default_rng(m + writes)
    # pairs (2k, 2k + 1) with k < n / 4: one member, one covered vertex; the rest isolated members
    k = np.arange(n // 4)
    nindex, nlist = W.csr_from_pairs(n, 2 * k, 2 * k + 1)
    mis = O.greedy_mis(nindex, nlist)
    orc = O.Oracle.from_csr(nindex, nlist)
    members = rng.permutation(np.nonzero(mis)[0])
    a, b = members[0:2 * writes:2], members[1:2 * writes:2]   # disjoint pairs of members
    short = writes - a.size
    extra = m - a.size
    u = np.concatenate([a, rng.choice(members, extra)])
    v = np.concatenate([b, rng.integers(0, n, extra)])
    assert short >= 0
    ok = u != v
    u, v = u[ok].astype(np.int32), v[ok].astype(np.int32)
    p = rng.permutation(u.size)
    u, v = u[p], v[p]
    with gb.Graph.from_csr(nindex, nlist) as g:
        for x in (g, orc):
            x.max_csr = 1 << 40
            x.set_mis(mis)
        for batch in range(2):
            ins = orc.flag_updates(u, v)
            g.apply_batch(u, v, ins)
            orc.apply_batch(u, v, ins)
            assert g.stats()["sub_batches"] == 1
            assert np.array_equal(g.get_mis(), orc.get_mis())
            assert np.array_equal(g.cluster_ids(), orc.cluster_ids())


def _greedy_graphs():
    yield "one", 1, *W.csr_from_pairs(2, [0], [1])
    for n in (31, 32, 33, 257, 3000):
        yield "path", n, *W.csr_from_pairs(n, np.arange(n - 1), np.arange(1, n))        # one chain through every tile
        yield "back", n, *W.csr_from_pairs(n, np.arange(n - 1), np.full(n - 1, n - 1))  # everything below one vertex
    yield "er", 20000, *W.er_graph(20000, 9, 3)
    yield "rmat", 4096, *W.rmat_graph(12, 12, 3)[1]


@pytest.mark.parametrize("kind,n,nindex,nlist", [pytest.param(*g, id="%s%d" % g[:2]) for g in _greedy_graphs()])
def test_greedy_passes(gb, kind, n, nindex, nlist):
    """The seed MIS of the base graph and of an evolved overlay, and the exact mode's completion (the same passes)."""
    import oracle as O
    orc = O.Oracle.from_csr(nindex, nlist)
    n = nindex.size - 1
    with gb.Graph.from_csr(nindex, nlist) as g:
        assert np.array_equal(g.greedy_mis(), O.greedy_mis(nindex, nlist))
        for x in (g, orc):
            x.set_mis(np.zeros(n, np.uint8))
            x.set_exact(True)
        rng = np.random.default_rng(n)
        m = min(400, 3 * n)
        for _ in range(2):
            u = rng.integers(0, n, m).astype(np.int32)
            v = ((u + rng.integers(1, max(n, 2), m)) % n).astype(np.int32)
            keep = u != v
            u, v = u[keep], v[keep]
            ins = rng.integers(0, 2, u.size).astype(np.uint8)
            g.apply_batch(u, v, ins)
            orc.apply_batch(u, v, ins)
            assert np.array_equal(g.get_mis(), orc.get_mis())
        orc.greedy_current()   # into the oracle's membership
        assert np.array_equal(g.greedy_mis(), orc.get_mis())


def test_parse_long_lines_over_read_chunks(gb, tmp_path):
    """Files longer than the read chunks, lines longer than a scan word, blank lines, no newline at the end."""
    rng = np.random.default_rng(1)
    with gb.Graph.from_csr(*W.er_graph(500, 6, 3)) as g:
        for size, tail in ((256 << 10, ""), (512 << 10, "\n"), ((768 << 10) + 5, "1 2")):
            parts, at = [], 0
            while at < size:
                kind = rng.integers(0, 4)
                a, b = rng.integers(0, 600, 2)
                line = ("%d %d" % (a, b), "%d\t%d %s" % (a, b, "x" * rng.integers(1, 200)), "", "%% %d" % a)[kind]
                parts.append(line)
                at += len(line) + 1
            path = str(tmp_path / "1.mtx")
            with open(path, "w") as f:
                f.write("\n".join(parts)[:size] + tail)
            u, v = gb.read_batch_file(path, 500)
            du, dv, di = g.parse_batch_file(path)
            assert u.size > 1000
            assert np.array_equal(du, u) and np.array_equal(dv, v) and np.array_equal(di, g.flag_updates(u, v))


@pytest.mark.parametrize("kind,m,max_csr,exact", [
    ("er", 600, 100000, False), ("er", 600, 100000, True),        # short rows, many sub-batches, growth on the way
    ("rmat", 800, 300000, False), ("rmat", 800, 300000, True),    # long rows
    ("sparse", 9000, 4000000, False),                             # sub-batches of 1,025 to 8,192 edges
    ("sparse", 30000, 30000000, False),                           # of more than 8,192 (assigned over the grid)
])
def test_overlapped_repairs(gb, kind, m, max_csr, exact):
    """Batches of several sub-batches without a trace, so that repairs overlap the next clustering; a batch refused in
    between changes nothing.  Membership, ids, limit and counters equal the oracle's, and the row map is left clean."""
    import oracle as O
    if kind == "er":
        nindex, nlist = W.er_graph(2000, 6, 5)
    elif kind == "rmat":
        nindex, nlist = W.rmat_graph(11, 8, 5)[1]
    else:
        nindex, nlist = W.er_graph(60000, 2, 5)
    n = nindex.size - 1
    mis = O.greedy_mis(nindex, nlist)
    orc = O.Oracle.from_csr(nindex, nlist)
    stream = W.ToggleStream(n, nindex, nlist, 6)
    subs = 0
    with gb.Graph.from_csr(nindex, nlist) as g:
        for x in (g, orc):
            x.max_csr = max_csr
            x.set_mis(mis)
            x.set_exact(exact)
        for k in range(3):
            u, v, ins = stream.next_batch(m, with_flags=True)
            g.apply_batch(u, v, ins)
            orc.apply_batch(u, v, ins)
            subs = max(subs, g.stats()["sub_batches"])
            assert np.array_equal(g.get_mis(), orc.get_mis()), k
            assert np.array_equal(g.cluster_ids(), orc.cluster_ids()), k
            assert g.max_csr == orc.max_csr
            bad = u.copy()
            bad[-1] = n
            with pytest.raises(gb.MisfitError):
                g.apply_batch(bad, v, ins)
            assert np.array_equal(g.get_mis(), orc.get_mis()) and np.array_equal(g.degrees(), orc.degrees())
    assert subs > 1


@pytest.mark.parametrize("zone", [30000, 1000])
def test_vertices_past_the_last_candidate_row(gb, zone):
    """A hub's row fills the sub-batch's 10^6 rows, so the neighbours of the other seeds (larger ids) have none, and
    what the hop-2 part of those seeds reads of them comes without a row."""
    import oracle as O
    leaves = 1020000
    n = leaves + 1 + zone
    zi, zl = W.er_graph(zone, 3, zone)
    lo, hi = W.undirected_pairs(zone, zi, zl)
    nindex, nlist = W.csr_from_pairs(n, np.concatenate([np.zeros(leaves, np.int64), lo + leaves + 1]),
                                     np.concatenate([np.arange(1, leaves + 1), hi + leaves + 1]))
    mis = O.greedy_mis(nindex, nlist)
    orc = O.Oracle.from_csr(nindex, nlist)
    stream = W.ToggleStream(zone, zi, zl, 3)
    with gb.Graph.from_csr(nindex, nlist) as g:
        for x in (g, orc):
            x.set_mis(mis)
        for k in range(4):
            u, v, ins = stream.next_batch(zone // 50, with_flags=True)
            u, v = u + leaves + 1, v + leaves + 1
            if k & 1:
                u = np.append(u, 0).astype(np.int32)
                v = np.append(v, leaves + k).astype(np.int32)
                ins = np.append(ins, 1).astype(np.uint8)
            g.apply_batch(u, v, ins)
            orc.apply_batch(u, v, ins)
            assert np.array_equal(g.get_mis(), orc.get_mis()), k
            assert np.array_equal(g.cluster_ids(), orc.cluster_ids()), k


@pytest.mark.parametrize("n", [(1 << 20) - 1, (1 << 20) + 1])
def test_pull_by_row_tails(gb, n):
    """From 2^20 vertices on the pull reads the rows' last entries first: rows shorter than a tail, tombstones at row
    ends, rows with none, one and many added entries."""
    import oracle as O
    nindex, nlist = W.er_graph(n, 5, 7)
    mis = O.greedy_mis(nindex, nlist)
    orc = O.Oracle.from_csr(nindex, nlist)
    rng = np.random.default_rng(n)
    full = np.flatnonzero(np.diff(nindex) > 0)
    with gb.Graph.from_csr(nindex, nlist) as g:
        g.set_tuning(cand_push=2)
        for x in (g, orc):
            x.set_mis(mis)
        for k in range(3):
            a = rng.choice(full, 3000, replace=False)
            last = nlist[nindex[a + 1] - 1]                       # deleted: the rows' last entries
            w = rng.integers(0, n, 2000)
            x = (w + 1 + rng.integers(0, n - 1, 2000)) % n        # added: anywhere,
            hubs = np.repeat(a[:20], 25)                          # and 25 to each of 20 rows
            y = (hubs + 1 + rng.integers(0, n - 1, hubs.size)) % n
            u = np.concatenate([a, w, hubs]).astype(np.int32)
            v = np.concatenate([last, x, y]).astype(np.int32)
            ins = np.concatenate([np.zeros(a.size), np.ones(w.size + hubs.size)]).astype(np.uint8)
            g.apply_batch(u, v, ins)
            orc.apply_batch(u, v, ins)
            assert np.array_equal(g.get_mis(), orc.get_mis()), k
            assert np.array_equal(g.cluster_ids(), orc.cluster_ids()), k


@pytest.mark.parametrize("m", [1, 700, 4096, 4097])
@pytest.mark.parametrize("skew", [1, 2, 3])
def test_device_lines_at_any_address(gb, m, skew):
    """Device arrays that start between two words: the lines are copied, not read in place."""
    import oracle as O
    import torch
    n = 3000
    nindex, nlist = W.er_graph(n, 6, 2)
    mis = O.greedy_mis(nindex, nlist)
    orc = O.Oracle.from_csr(nindex, nlist)
    stream = W.ToggleStream(n, nindex, nlist, m)
    with gb.Graph.from_csr(nindex, nlist) as g:
        for x in (g, orc):
            x.set_mis(mis)
        for _ in range(2):
            u, v, ins = stream.next_batch(m, with_flags=True)
            raw = [np.zeros(a.nbytes + skew, np.uint8) for a in (u, v, ins)]
            for r, a in zip(raw, (u, v, ins)):
                r[skew:] = a.view(np.uint8)
            dev = [torch.as_tensor(r, device="cuda") for r in raw]
            torch.cuda.synchronize()
            g.apply_batch_device(*(d.data_ptr() + skew for d in dev), u.size)
            orc.apply_batch(u, v, ins)
            assert np.array_equal(g.get_mis(), orc.get_mis())
            assert np.array_equal(g.cluster_ids(), orc.cluster_ids())
            assert np.array_equal(g.degrees(), orc.degrees())


def test_overlapped_repairs_of_several_contexts(gb):
    """Batches of several sub-batches on eight contexts from eight threads at once, each batch larger than the last
    (buffers grow while other contexts hold the same side streams), contexts closing while others go on.  Every
    graph's membership, ids and limit equal its own oracle's."""
    from concurrent.futures import ThreadPoolExecutor
    import oracle as O

    def work(k):
        # (vertices, degree, lines, limit): short rows, long rows, fronts on a side stream, host-driven rounds
        n, degree, sizes, limit = ((3000, 6, (200, 600, 1200), 150000), (None, 8, (300, 700, 1100), 400000),
                                   (70000, 4, (3000, 6000, 9000), 4000000),
                                   (70000, 2, (20000, 60000, 90000), 120000000))[k % 4]
        nindex, nlist = W.rmat_graph(11, degree, k)[1] if n is None else W.er_graph(n, degree, k)
        n = nindex.size - 1
        mis = O.greedy_mis(nindex, nlist)
        orc = O.Oracle.from_csr(nindex, nlist)
        stream = W.ToggleStream(n, nindex, nlist, k)
        subs = 0
        with gb.Graph.from_csr(nindex, nlist) as g:
            for x in (g, orc):
                x.max_csr = limit
                x.set_mis(mis)
            for m in sizes:
                u, v, ins = stream.next_batch(m, with_flags=True)
                g.apply_batch(u, v, ins)
                orc.apply_batch(u, v, ins)
                subs = max(subs, g.stats()["sub_batches"])
                assert np.array_equal(g.get_mis(), orc.get_mis()), (k, m)
                assert np.array_equal(g.cluster_ids(), orc.cluster_ids()), (k, m)
                assert g.max_csr == orc.max_csr, (k, m)
        return subs

    with ThreadPoolExecutor(8) as pool:
        assert min(pool.map(work, range(16))) > 1


@pytest.mark.parametrize("mb", [2, 12])
def test_parsing_gives_its_text_back(gb, tmp_path, mb):
    """After a batch file the context holds its lines, nine bytes each, and for files up to 4 MB the text and line
    starts; not nine bytes for each byte of a large file."""
    import ctypes
    lines = mb * 100000
    rng = np.random.default_rng(mb)
    u, v = rng.integers(1000000, 2000000, (2, lines))
    path = str(tmp_path / "1.mtx")
    with open(path, "w") as f:
        f.write("".join("%07d %07d padded\n" % p for p in zip(u, v)))
    rt = ctypes.CDLL({l.split()[-1] for l in open("/proc/self/maps") if "libcudart" in l}.pop())
    with gb.Graph.from_csr(*W.er_graph(1000, 4, 1)) as g:
        pool, used = ctypes.c_void_p(), [ctypes.c_uint64(), ctypes.c_uint64()]
        assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
        assert rt.cudaMemPoolGetAttribute(pool, 7, ctypes.byref(used[0])) == 0   # cudaMemPoolAttrUsedMemCurrent
        assert g.parse_batch_file(path)[0].size == 0    # ids past the graph: every line is read, none kept
        assert rt.cudaMemPoolGetAttribute(pool, 7, ctypes.byref(used[1])) == 0
    held = used[1].value - used[0].value
    assert held <= 9 * lines + (1 << 20) + (9 * 23 * lines if mb <= 4 else 0)


@pytest.fixture(scope="module", params=[0, 300])
def crowded(request):
    """A graph and two batches of one sub-batch each whose seeds leave fewer rows than there are candidates (a
    sub-batch has 2^21 rows), all rows short or one of them long; and what the oracle gives."""
    import oracle as O
    n, m = 3000000, 1040000
    rng = np.random.default_rng(1)
    a, b = rng.integers(0, n, (2, int(1.2 * n)))
    a[:request.param] = 7
    ok = a != b
    nindex, nlist = W.csr_from_pairs(n, a[ok], b[ok])
    orc = O.Oracle.from_csr(nindex, nlist)
    mis = O.greedy_mis(nindex, nlist)
    orc.max_csr = 1 << 40
    orc.set_mis(mis)
    batches, want = [], []
    for _ in range(2):
        u = rng.integers(0, n, m).astype(np.int32)
        v = ((u + rng.integers(1, n, m)) % n).astype(np.int32)
        batches.append((u, v, (rng.random(m) < 0.9).astype(np.uint8)))
        orc.apply_batch(*batches[-1])
        want.append((orc.get_mis(), orc.cluster_ids()))
    return nindex, nlist, mis, batches, want


@pytest.mark.parametrize("push", [1, 2])
def test_more_candidates_than_rows(gb, crowded, push):
    """Hop-1 vertices past the last candidate row have no row: the hop-2 part reads theirs again (short rows) or
    searches them for their ids alone, and their tag bits outlive the sub-batch."""
    nindex, nlist, mis, batches, want = crowded
    with gb.Graph.from_csr(nindex, nlist) as g:
        g.max_csr = 1 << 40
        g.set_mis(mis)
        g.set_tuning(cand_push=push)
        for (u, v, ins), (members, ids) in zip(batches, want):
            g.apply_batch(u, v, ins)
            st = g.stats()
            assert st["sub_batches"] == 1 and st["seeds"] + st["candidates"] == 1 << 21   # every row is taken
            assert np.array_equal(g.get_mis(), members)
            assert np.array_equal(g.cluster_ids(), ids)


@pytest.mark.parametrize("m", [40, 5000])
@pytest.mark.parametrize("shuffled", [False, True])
def test_pairs_of_many_updates(gb, m, shuffled):
    """One to eleven updates of a pair in a batch (the first apart, then four at a time), both directions and every
    flag, on rows with repeated entries, sorted or not; and one pair for the whole batch."""
    import oracle as O
    n = 900
    rng = np.random.default_rng(m)
    a, b = rng.integers(0, n, (2, 4000))
    a[:200], b[:200] = 5, rng.integers(6, 60, 200)        # a hub whose row repeats its entries
    ok = a != b
    x, y = np.concatenate([a[ok], b[ok]]), np.concatenate([b[ok], a[ok]])
    order = np.lexsort((rng.random(x.size) if shuffled else y, x))
    nlist = y[order].astype(np.int32)
    nindex = np.concatenate([[0], np.cumsum(np.bincount(x, minlength=n))]).astype(np.int64)
    mis = O.greedy_mis(nindex, nlist)
    orc = O.Oracle.from_csr(nindex, nlist)
    with gb.Graph.from_csr(nindex, nlist) as g:
        for z in (g, orc):
            z.set_mis(mis)
        for batch in range(4):
            if batch == 2:
                u, v = np.full(m, 5), np.full(m, 7)
            else:
                pairs = np.concatenate([np.full((m, 1), 5), rng.integers(6, 60, (m, 1))], 1)
                far = rng.random(m) < 0.5
                pairs[far] = rng.integers(0, n, (far.sum(), 2))
                pairs = np.repeat(pairs, rng.integers(1, 12, m), axis=0)
                pairs = pairs[pairs[:, 0] != pairs[:, 1]][:m]
                u, v = pairs[rng.permutation(len(pairs))].T
            flip = rng.random(u.size) < 0.5
            u, v = np.where(flip, v, u).astype(np.int32), np.where(flip, u, v).astype(np.int32)
            ins = rng.integers(0, 2, u.size).astype(np.uint8)
            g.apply_batch(u, v, ins)
            orc.apply_batch(u, v, ins)
            assert np.array_equal(g.degrees(), orc.degrees()), batch
            for z in range(0, n, 7):
                assert np.array_equal(g.row(z), orc.row(z)), (batch, z)
            assert np.array_equal(g.row(5), orc.row(5)), batch
            assert np.array_equal(g.get_mis(), orc.get_mis()), batch
            assert np.array_equal(g.cluster_ids(), orc.cluster_ids()), batch


@pytest.mark.parametrize("n", [(1 << 20) - 1, 1 << 20])
def test_pull_bytes_of_the_profile(gb, n):
    """By row tails 32 B a vertex and nothing twice; by the bounds 28 B and four for each row entry looked at."""
    nindex, nlist = W.er_graph(n, 5, 7)
    with gb.Graph.from_csr(nindex, nlist) as g:
        g.set_tuning(cand_push=2)
        g.set_mis(g.greedy_mis())
        g.profile(1)
        g.apply_batch(*W.ToggleStream(n, nindex, nlist, 3).next_batch(2000, with_flags=True))
        _, calls, nbytes = g.profile_read()["pull"]
    assert calls > 0
    if n >= 1 << 20:
        assert nbytes == 32.0 * n * calls
    else:
        assert 28.0 * n * calls < nbytes < (28.0 * n + 4.0 * nlist.size) * calls
