"""A closed basin started hours before time 0 (GPU): no edge is open, so no boundary table is
read, and the steps are those of the same basin started at 0, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t_start", [-3600.0, -7200.0, -3.6e6])
def test_closed_basin_before_time_zero(t_start):
    from hydist import cases
    from hydist.lib import Simulation
    c = cases.channel_case(N=40, M=36, dX=5.0, dT=2.0, bank=4, slope=0.0, hours=1)
    c.fields["h"][:6, :] = c.fields["h"][0, 0]  # dry banks across both ends too
    c.fields["h"][-6:, :] = c.fields["h"][0, 0]
    c.fields["z"][18:22, :] += 0.1
    c.boundary_type[:] = 0
    out = []
    for t in (0.0, t_start):
        c.t_start = t
        s = Simulation.from_case(c)
        s.step(30)
        for f in ("moci", "mocj"):  # the lines the edges' values go to
            m = s.get(f)
            assert m[2] == 0 and m[s.N if f == "moci" else s.M] == 0
        out.append({f: s.get(f) for f in ("z", "u", "v", "khouot")})
        s.close()
    assert np.isfinite(out[0]["z"]).all() and np.abs(out[0]["u"]).max() > 0
    for f, a in out[0].items():
        assert np.array_equal(a, out[1][f]), f
