"""A batch that runs out of device memory: it has changed nothing, or its links
are all in the graph; either way the context goes on as if it had been made
in that state.  Every allocation of a context's first batch is refused in
turn (MISFIT_GB_FAIL_ALLOC, on the host).  All values are integers or bytes:
comparisons are exact."""
import numpy as np
import pytest

import oracle as O
from misfit_gb300 import native
from misfit_gb300 import workloads as W

pytestmark = pytest.mark.gpu

ENOMEM = -5


def _case(kind):
    if kind == "short":        # one sub-batch of short rows
        nindex, nlist = W.er_graph(3000, 6, 5)
        return nindex, nlist, 300, 0, 0
    if kind == "short_pull":   # the same by the pull
        nindex, nlist = W.er_graph(3000, 6, 5)
        return nindex, nlist, 300, 0, 2
    if kind == "long":         # rows of any length, one sub-batch
        nindex, nlist = W.rmat_graph(11, 8, 5)[1]
        return nindex, nlist, 100, 1 << 40, 0
    if kind == "many":         # several sub-batches: overlapped repairs, exact sizes, growth on the way
        nindex, nlist = W.er_graph(2000, 6, 5)
        return nindex, nlist, 600, 100000, 0
    nindex, nlist = W.er_graph(60000, 2, 5)   # "wide": more than one block plans and sorts, commits by a large block
    return nindex, nlist, 9000, 4000000, 0


@pytest.mark.parametrize("kind", ["short", "short_pull", "long", "many", "wide"])
def test_every_refused_allocation(gpu_lib, monkeypatch, kind):
    nindex, nlist, m, max_csr, push = _case(kind)
    n = nindex.size - 1
    mis0 = O.greedy_mis(nindex, nlist)
    stream = W.ToggleStream(n, nindex, nlist, 6)
    first = stream.next_batch(m, with_flags=True)
    probe = np.unique(first[0])[:40]

    def oracle_at(after, mis, limit):
        orc = O.Oracle.from_csr(nindex, nlist)
        if after:
            orc.apply_overlay(*first)
        orc.set_mis(mis)
        orc.max_csr = limit
        return orc

    whole = O.Oracle.from_csr(nindex, nlist)
    if max_csr:
        whole.max_csr = max_csr
    whole.set_mis(mis0)
    whole.apply_batch(*first)
    k, before, after = 0, 0, 0
    while True:
        k += 1
        monkeypatch.setenv("MISFIT_GB_FAIL_ALLOC", str(k))
        with native.Graph.from_csr(nindex, nlist) as g:
            if push:
                g.set_tuning(cand_push=push)
            if max_csr:
                g.max_csr = max_csr
            g.set_mis(mis0)
            try:
                g.apply_batch(*first)
                break   # its first batch makes fewer allocations than k
            except native.MisfitError as e:
                assert e.status == ENOMEM, k
            mis = g.get_mis()
            assert mis.max() <= 1, k
            done = not np.array_equal(g.degrees(), np.diff(nindex))
            orc = oracle_at(done, mis, g.max_csr)
            assert np.array_equal(g.degrees(), orc.degrees()), k
            for x in probe:
                assert np.array_equal(g.row(int(x)), orc.row(int(x))), (k, x)
            ids = g.cluster_ids()
            if done:
                after += 1
                if kind not in ("many", "wide"):   # one sub-batch: its clustering ran or did not, its repair did not
                    assert np.all(ids == -1) or np.array_equal(ids, whole.cluster_ids()), k
                    assert np.array_equal(mis, mis0), k
            else:
                before += 1
                assert np.all(ids == -1) and np.array_equal(mis, mis0), k
            g.set_mis(mis)   # ids of both sides to none
            u, v = stream.next_batch(m // 2)
            for batch in range(2):
                ins = orc.flag_updates(u, v)
                g.apply_batch(u, v, ins)
                orc.apply_batch(u, v, ins)
                assert np.array_equal(g.get_mis(), orc.get_mis()), (k, batch)
                assert np.array_equal(g.cluster_ids(), orc.cluster_ids()), (k, batch)
                assert np.array_equal(g.degrees(), orc.degrees()), (k, batch)
                assert g.max_csr == orc.max_csr, (k, batch)
    assert before > 5 and after > 3, (before, after)


@pytest.mark.parametrize("kind", ["short", "long", "wide"])
def test_first_batch_allocates_in_groups(gpu_lib, kind):
    """A context's first batch needs some seventy buffers; an allocation is the dearer the more contexts the device has
    had, so buffers that grow together are parts of one (three groups of the batch's, the graph's and the repair's
    size, and what each path adds)."""
    nindex, nlist, m, max_csr, _ = _case(kind)
    with native.Graph.from_csr(nindex, nlist) as g:
        if max_csr:
            g.max_csr = max_csr
        g.set_mis(O.greedy_mis(nindex, nlist))
        before = native.allocations()
        g.apply_batch(*W.ToggleStream(nindex.size - 1, nindex, nlist, 6).next_batch(m, with_flags=True))
        assert native.allocations() - before <= 40


@pytest.mark.parametrize("kind", ["short", "long", "many", "wide"])
def test_refused_allocations_of_a_later_larger_batch(gpu_lib, monkeypatch, kind):
    """The same for the second batch of a context, three times the first: its buffers grow, and what must be zero or
    mapped nowhere between batches stands in some of them."""
    nindex, nlist, m, max_csr, push = _case(kind)
    n = nindex.size - 1
    mis0 = O.greedy_mis(nindex, nlist)
    stream = W.ToggleStream(n, nindex, nlist, 7)
    small = stream.next_batch(m // 3, with_flags=True)
    large = stream.next_batch(m, with_flags=True)
    u, v = stream.next_batch(m // 2)

    def start(x):
        if max_csr:
            x.max_csr = max_csr
        x.set_mis(mis0)
        x.apply_batch(*small)

    monkeypatch.delenv("MISFIT_GB_FAIL_ALLOC", raising=False)
    with native.Graph.from_csr(nindex, nlist) as g:
        opened = native.allocations()
        start(g)
        k = native.allocations() - opened - 4   # the first batch's, some of which do not count for the refusal
    refused = 0
    while True:
        k += 1
        monkeypatch.setenv("MISFIT_GB_FAIL_ALLOC", str(k))
        with native.Graph.from_csr(nindex, nlist) as g:
            try:
                start(g)
            except native.MisfitError:
                continue   # still the first batch's
            degrees = g.degrees()
            try:
                g.apply_batch(*large)
                break
            except native.MisfitError as e:
                assert e.status == ENOMEM, k
            refused += 1
            mis = g.get_mis()
            assert mis.max() <= 1, k
            orc = O.Oracle.from_csr(nindex, nlist)
            start(orc)
            if not np.array_equal(g.degrees(), degrees):
                orc.apply_overlay(*large)
            else:
                assert np.array_equal(mis, orc.get_mis()) and np.array_equal(g.cluster_ids(), orc.cluster_ids()), k
            assert np.array_equal(g.degrees(), orc.degrees()), k
            orc.set_mis(mis)
            orc.max_csr = g.max_csr
            g.set_mis(mis)
            for batch in range(2):
                ins = orc.flag_updates(u, v)
                g.apply_batch(u, v, ins)
                orc.apply_batch(u, v, ins)
                assert np.array_equal(g.get_mis(), orc.get_mis()), (k, batch)
                assert np.array_equal(g.cluster_ids(), orc.cluster_ids()), (k, batch)
                assert np.array_equal(g.degrees(), orc.degrees()), (k, batch)
    assert refused > 3
