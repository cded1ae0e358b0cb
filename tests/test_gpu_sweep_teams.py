"""The line sweeps' teams (GPU): a line's values are the same bits whichever warps sweep it.

One reach whose rows are short, whose columns are long and whose island lines have several
segments, stepped with launch shapes that give a CTA a few lines or a hundred, in one round
or in many (more rows than the shared memory holds at once), in both precisions.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("z", "u", "v", "FS", "dH", "khouot")


def _run(case, shape, n):
    from hydist.lib import Simulation
    sim = Simulation.from_case(case)
    if shape:
        sim.set_sweep_shape(*shape)
    sim.step(n)
    out = {f: sim.get(f) for f in FIELDS}
    sim.close()
    return out


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("N,M", [(700, 90), (90, 700), (260, 250)])
def test_shapes_give_the_same_bits(N, M, mixed):
    from hydist import cases
    c = cases.islands_case(N=N, M=M, seed=5)
    p = c.params.copy()
    p.precision_mode = mixed
    c.params = p
    ref = _run(c, None, 25)
    assert np.isfinite(ref["z"]).all()
    for shape in ((1, 0), (1, 1), (5, 0), (40, 1)):
        got = _run(c, shape, 25)
        for f in FIELDS:
            assert np.array_equal(got[f], ref[f], equal_nan=f != "khouot"), (shape, f)
