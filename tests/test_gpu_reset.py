"""A process that closes its contexts, resets the device and opens new ones:
nothing that the library keeps for the process may belong to the old device
context.  Run in a child process; the values are compared with the oracle's."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import oracle as O
from misfit_gb300 import native
from misfit_gb300 import workloads as W

kind = sys.argv[2]
n, degree, m, max_csr = {"lines": (3000, 6, 3000, 1 << 40), "edges": (60000, 2, 6000, 1 << 40),
                         "overlap": (80000, 4, 4000, 3000000)}[kind]
nindex, nlist = W.er_graph(n, degree, 3)
mis = O.greedy_mis(nindex, nlist)
native.load_library()
libs = {l.split()[-1] for l in open("/proc/self/maps") if "libcudart" in l}
assert len(libs) == 1, libs
reset = ctypes.CDLL(libs.pop()).cudaDeviceReset
for life in range(3):
    orc = O.Oracle.from_csr(nindex, nlist)
    stream = W.ToggleStream(n, nindex, nlist, 4)
    with native.Graph.from_csr(nindex, nlist) as g:
        for x in (g, orc):
            x.max_csr = max_csr
            x.set_mis(mis)
        for batch in range(2):
            u, v, ins = stream.next_batch(m, with_flags=True)
            g.apply_batch(u, v, ins)
            orc.apply_batch(u, v, ins)
            assert np.array_equal(g.get_mis(), orc.get_mis()), (life, batch)
            assert np.array_equal(g.cluster_ids(), orc.cluster_ids()), (life, batch)
            assert (g.stats()["sub_batches"] > 1) == (kind == "overlap")
    assert reset() == 0
print("ok")
"""


@pytest.mark.parametrize("kind", ["lines", "edges", "overlap"])
def test_new_contexts_after_a_device_reset(gpu_lib, kind):
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, kind], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split() == ["ok"], r.stderr[-2000:]
