"""The steady residual's snapshot holds every cell that can be wet, dry ones too (GPU): a cell that
opens after the snapshot is compared with what stood there at the snapshot, not with an earlier
snapshot's or no value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("earlier", [False, True])
def test_cell_opened_after_the_snapshot(earlier):
    from hydist import cases
    from hydist.lib import Simulation
    sim = Simulation.from_case(cases.islands_case())
    sim.step(20)
    kh = sim.get("khouot")
    wet = np.argwhere(kh[2:sim.N + 1, 2:sim.M + 1] == 0) + 2
    cells = tuple(wet[:: len(wet) // 7].T)  # a few cells all over the reach
    if earlier:
        sim.steady_residual(snapshot=True)  # with the cells wet
    closed = kh.copy()
    closed[cells] = 1
    at = {f: sim.get(f) for f in ("u", "v", "z")}
    for k, f in enumerate(("u", "v", "z")):
        at[f][cells] += 0.5 + k  # what stands there at the snapshot
        sim.set(f, at[f])
    sim.set("khouot", closed)
    sim.steady_residual(snapshot=True)
    sim.set("khouot", kh)
    now = {f: a + 0.01 for f, a in at.items()}
    for f, a in now.items():
        sim.set(f, a)
    r = sim.steady_residual(snapshot=False)
    w = np.zeros_like(kh, dtype=bool)
    w[2:sim.N + 1, 2:sim.M + 1] = kh[2:sim.N + 1, 2:sim.M + 1] == 0
    d = {f: (now[f] - at[f])[w] for f in now}
    H = sim.get("H_moi")[w]
    mom = np.sqrt((d["u"] ** 2 + d["v"] ** 2).sum() / (now["u"][w] ** 2 + now["v"][w] ** 2).sum())
    con = np.sqrt((d["z"] ** 2).sum() / (H ** 2).sum())
    assert abs(r[0] - mom) <= 1e-12 * mom and abs(r[1] - con) <= 1e-12 * con, (r, mom, con)
    sim.close()
