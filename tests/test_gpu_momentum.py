"""The explicit momentum cell by cell (GPU) against the form that walks the segment tables
line by line: the same bits, on reaches with one- and two-cell segments, segments on every
edge of the grid, and every edge open or a wall.

The second simulation has a segment table set (to what it is) before every step, which makes
the step rescan every line and take whole-grid passes and the table-driven kernels.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("z", "u", "v", "t_u", "t_v", "FS", "khouot")


def _turned(c):
    """The reach with x and y exchanged: its open edges become the down and up edges."""
    from hydist import cases
    d = cases.islands_case(N=c.N, M=c.M, seed=c.notes["seed"])
    d.N, d.M = c.M, c.N
    d.fields = {f: np.ascontiguousarray(c.fields[f].T) for f in cases.GRID_FIELDS}
    d.boundary_type = np.zeros_like(c.boundary_type)
    d.boundary_type[cases.EDGE_DOWN, 0] = 2
    d.boundary_type[cases.EDGE_UP, 0] = 1
    z = np.zeros((1, c.total_time))
    d.tables = [c.tables[3], c.tables[2], z, z]
    d.cc = [c.cc[3], c.cc[2], z, z]
    return d


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("turn", [False, True])
@pytest.mark.parametrize("N,M,seed", [(48, 36, 7), (33, 80, 5), (97, 140, 3)])
def test_cells_match_lines(N, M, seed, turn, mixed):
    from hydist import cases
    from hydist.lib import Simulation
    c = cases.islands_case(N=N, M=M, seed=seed)
    if turn:
        c = _turned(c)
    p = c.params.copy()
    p.precision_mode = mixed
    c.params = p
    a, b = Simulation.from_case(c), Simulation.from_case(c)
    for k in range(40):
        b.set("moci", b.get("moci"))
        a.step(1)
        b.step(1)
        if k % 8 == 7:
            for f in FIELDS:
                assert np.array_equal(a.get(f), b.get(f)), (k, f)
    a.close()
    b.close()
