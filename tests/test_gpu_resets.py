"""The wet/dry resets (GPU) against the oracle where their shapes change: a column by one warp
alone or four to a CTA (the last CTA partly empty), columns of one load per lane, of two and
of a second round, and rows of more words than a warp has lanes.

Every fourth step starts from disturbed levels, so that runs of dry cells open in cascades (across
words too) and wet cells close; fields, mask and segment tables are compared.  The lines are
solved serially: a cell opens when its new level is above the old one, and where they are equal
but for rounding only the oracle's order of elimination decides as the oracle does.
"""
import numpy as np
import pytest

from helpers import EXACT_FIELDS, compare

pytestmark = pytest.mark.gpu

FIELDS = ("z", "t_z", "t_u", "t_v", "FS", "H_moi")


@pytest.mark.parametrize("N,M", [(40, 594), (530, 34), (1100, 30), (30, 1100)])
def test_resets_vs_oracle(oracle_lib, N, M, monkeypatch):
    import oracle
    from hydist import cases
    from hydist.lib import Simulation
    monkeypatch.setenv("HYD_SOLVER", "thomas")
    c = cases.islands_case(N=N, M=M, seed=11)
    sim = Simulation.from_case(c)
    ora = oracle.OracleSim(c)
    ora.init()
    rng = np.random.default_rng(N + M)
    for k in range(8):
        if k % 4 == 0:
            z = ora.get("z")
            z = np.where(ora.get("khouot") == 0, z + 0.05 * rng.standard_normal(z.shape), z)
            sim.set("z", z)
            ora.view("z")[...] = z
        sim.step(1)
        ora.step(1)
        assert max(ora.get("moci").max(), ora.get("mocj").max()) < 20
        compare(sim, ora.get, fields=FIELDS, exact=EXACT_FIELDS)
    sim.close()
