"""The tuner tries the shape a batch starts with (GPU), whichever its number of lines chose."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,N,M", [(2, 60, 40), (12, 400, 60), (20, 400, 60), (40, 300, 60), (3, 900, 40)])
def test_starting_shape_is_a_candidate(count, N, M):
    from hydist import cases
    from hydist.lib import Batch
    from hydist.tune import DEFAULT_CANDIDATES, FUSED, apply_policy
    batch = Batch([cases.channel_case(N=N, M=M)] * count)
    start = [m.sweep_shape() for m in batch.members]
    tried = []
    for policy in DEFAULT_CANDIDATES:
        if policy != FUSED:
            apply_policy(batch, policy)
            tried.append([m.sweep_shape() for m in batch.members])
    batch.close()
    assert start in tried, (start[0], [t[0] for t in tried])
