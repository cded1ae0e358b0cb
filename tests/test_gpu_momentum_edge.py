"""The open edge's face where the edge's first wet segment is one cell: it is extrapolated from
the velocities that stood on faces 2 and 3, also where the next segment starts at cell 4 and its
wall end puts 0 on face 3 in the same pass.

A closed pair of cells keeps a velocity on the face between them (a caller's: the model's own
states leave 0 there), and the cell beyond opens on its own while the reach steps, so that the
line reads [2, 2] wet, 3 dry, [4, 4] wet with that velocity still on face 3.
"""
import numpy as np
import pytest

J0 = 9        # the line of the pattern
V0 = 0.4      # the velocity between the closed cells
STEPS = 12
FIELDS = ("z", "u", "v", "t_u", "t_v", "khouot")


def _case(turn):
    """A straight reach with its discharge edge at i = 2 (turned: at j = 2), the level low by 0.2 m
    over some rows beyond the pattern: it falls at first and rises within a few steps."""
    from hydist import cases
    c = cases.channel_case(N=24, M=20, dX=5.0, dT=1.0, bank=2, depth=3.0, slope=0.0, Q=20.0, hours=1, z_out=0.0)
    c.fields["z"][6:12, :] -= 0.2
    if turn:
        c.N, c.M = c.M, c.N
        c.fields = {f: np.ascontiguousarray(c.fields[f].T) for f in cases.GRID_FIELDS}
        c.boundary_type = np.zeros_like(c.boundary_type)
        c.boundary_type[cases.EDGE_DOWN, 0] = 2
        c.boundary_type[cases.EDGE_UP, 0] = 1
        z = np.zeros((1, c.total_time))
        c.tables, c.cc = [c.tables[3], c.tables[2], z, z], [c.cc[3], c.cc[2], z, z]
    return c


def _turned(a, turn):
    return a.T if turn else a


def _oracle(c, turn):
    import oracle
    o = oracle.OracleSim(c)
    o.init()
    mask = o.get("khouot")
    m = _turned(mask, turn)
    m[3, J0], m[4, J0], m[5, J0] = 2, 1, 2
    vel = np.zeros_like(o.get("t_u"))
    _turned(vel, turn)[3, J0] = V0
    p = oracle.OracleSim(c)
    p.view("khouot")[...] = mask
    p.init_pickup()
    p.view("t_v" if turn else "t_u")[...] = vel
    return p, mask, vel


@pytest.mark.parametrize("turn", [0, 1])
def test_case_reaches_the_pattern(oracle_lib, turn):
    """On the CPU: cell 4 opens after the first step, alone between dry cells, beside a one-cell
    segment at the edge, and the edge's face takes the velocity that stood on face 3."""
    o, _, _ = _oracle(_case(turn), turn)
    t = "t_v" if turn else "t_u"
    seen = 0
    for n in range(STEPS):
        mask0, face3 = _turned(o.get("khouot"), turn)[2:6, J0].tolist(), _turned(o.get(t), turn)[3, J0]
        o.step(1)
        mask1, vel1 = _turned(o.get("khouot"), turn)[2:6, J0].tolist(), _turned(o.get(t), turn)[:, J0]
        # u: the cell opens between the half-steps; v: before the step
        if n > 0 and (mask0 if turn else mask1) == [0, 2, 0, 2] and face3 != 0.0:
            seen += 1
            assert vel1[3] == 0.0 and abs(vel1[1]) > 0.1
    assert seen == 1


@pytest.mark.gpu
@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("turn", [0, 1])
def test_edge_face_reads_before_it_is_written(oracle_lib, turn, mixed):
    """Cell by cell against the segment tables line by line (a table set before every step): the
    same bits."""
    from hydist.lib import Simulation
    c = _case(turn)
    _, mask, vel = _oracle(c, turn)
    p = c.params.copy()
    p.precision_mode = mixed
    c.params = p
    sims = []
    for _ in range(2):
        s = Simulation.from_case(c, init=False)
        s.set("khouot", mask)
        s.init_pickup()
        s.set("t_v" if turn else "t_u", vel)
        sims.append(s)
    a, b = sims
    for n in range(STEPS):
        b.set("moci", b.get("moci"))
        a.step(1)
        b.step(1)
        for f in FIELDS:
            assert np.array_equal(a.get(f), b.get(f)), (n, f)
    a.close()
    b.close()
