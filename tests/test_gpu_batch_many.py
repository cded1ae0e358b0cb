"""Batched launches with more members than a warp has lanes (GPU): a CTA finds its member among
lists of 33 and of 70, and every member ends with the bits of the same batch stepped member by
member."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("z", "u", "v", "t_z", "t_u", "t_v", "FS", "dH", "khouot", "daui", "cuoii", "moci", "dauj", "cuoij", "mocj")


@pytest.mark.parametrize("count", [32, 33, 70])
def test_many_members(count):
    from hydist import cases
    from hydist.lib import Batch
    cs = [cases.islands_case(N=30 + (7 * k) % 41, M=28 + (11 * k) % 29, seed=k) for k in range(count)]
    a, b = Batch(cs), Batch(cs)
    a.set_fused(True)
    a.step(30)
    b.step(30)
    assert a.fused_steps() >= 25
    for k, (ma, mb) in enumerate(zip(a.members, b.members)):
        for f in FIELDS:
            assert np.array_equal(ma.get(f), mb.get(f), equal_nan=True), (k, f)
    a.close()
    b.close()
