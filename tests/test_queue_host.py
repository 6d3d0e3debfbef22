"""The number of steps queued before the host looks for a collider request (CPU): up to where the last interval ended,
and soon as many as allowed again once the runs stay out."""
import pytest

from woodem_gb300 import _native


@pytest.mark.parametrize("most", [1, 2, 32, 1024])
@pytest.mark.parametrize("interval", [0, 1, 2, 3, 8, 40, 5000])
def test_chunks(most, interval, gpu_lib):
    q = _native.lib().wg_steps_to_queue
    since = waits = 0
    while since < 100000:
        k = q(most, since, interval)
        assert 1 <= k <= most
        if interval and since < interval:
            assert k == min(most, interval + 1 - since)
        since, waits = since + k, waits + 1
    # at rest: as many waits as the steps need, and about four for each doubling on the way there
    assert q(most, since, interval) == most
    assert waits <= 100000 / most + 2 * 4 * 17 + 4
