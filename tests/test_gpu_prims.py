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
