"""Event counts of k_resident over steps that are replayed: every committed
step's zeroth-, first- and second-order events count once, whatever step of a
launch fails.  Whole numbers, so there is no tolerance."""
import pytest

from test_gpu_parity import run_parity
from test_gpu_resident import system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [5, 6, 7])
@pytest.mark.parametrize("kon,capacity", [(2.0, 0), (0.5, 1500), (8.0, 0)])
def test_event_counts_across_replayed_steps(kon, capacity, seed):
    """Births fill the cells past their bins (and, with a capacity given, the
    slots) again and again in the middle of launches whose steps have
    candidate pairs."""
    s = system(50, 6, kon=kon, births=60.0, seed=seed, capacity=capacity)
    assert s.kernels_per_step() == 1
    _, pairs, events = run_parity(s, 60, batch=60)
    assert pairs > 0 and all(events > 0)
    s.close()
