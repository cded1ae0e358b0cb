"""hyd_set_sweep_shape changes the line sweeps' launch shape only (GPU): a step's launches are as
many whatever the shape, for a reach alone on the device and for a batch's members, whose steps
leave the smoothing apart from the explicit momentum."""
import pytest

pytestmark = pytest.mark.gpu


def _launches(sim, step):
    step(2)  # the whole-grid step, and the graph of the steps that follow
    a = sim.launch_count()
    step(1)
    return sim.launch_count() - a


def test_launches_do_not_depend_on_the_shape():
    from hydist import cases
    from hydist.lib import Batch, Simulation
    c = cases.channel_case(N=100, M=40)
    sim = Simulation.from_case(c)
    alone = []
    for ctas, wide in ((0, 0), (0, 1), (4, 0), (4, 1)):
        sim.set_sweep_shape(ctas, wide)
        alone.append(_launches(sim, sim.step))
    sim.close()
    batch = Batch([c, c])
    member = []
    for ctas, wide in ((4, 1), (4, 0), (8, 1), (8, 0)):
        for m in batch.members:
            m.set_sweep_shape(ctas, wide)
        member.append(_launches(batch.members[0], batch.step))
    batch.close()
    assert len(set(alone)) == 1 and len(set(member)) == 1, (alone, member)
    assert member[0] == 2 * (alone[0] + 2), (alone, member)  # two members, two smoothing launches more each
