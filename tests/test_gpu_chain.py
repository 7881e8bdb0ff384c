"""The kernel chain of the binned sort (k_bin, k_scan, k_pairs_cells,
k_pairs_big, k_match) on grids of more cells than k_resident takes, GPU
against the oracle bit for bit.  Bits are compared, so there is no
tolerance."""
import numpy as np
import pytest

from gpusmoldyn_gb300.configs import rng, uniform_positions
from test_gpu_parity import run_parity
from test_gpu_resident import system

pytestmark = pytest.mark.gpu

CELLS = 54  # 157,464 cells of edge 0.25


@pytest.mark.parametrize("births", [0.7, 40.0, 2000.0])
def test_bins_overflow_beside_births_in_the_last_cta(births):
    """A cluster overflows its bin while the last CTA of k_bin makes the
    step's births: the step stops whole and is replayed with larger bins."""
    s = system(3000, CELLS, births=births)
    g = rng(17)
    pos = uniform_positions(g, 3000, (0, 0, 0), (0.25 * CELLS,) * 3)
    pos[:400] = uniform_positions(g, 400, (0.3,) * 3, (0.4,) * 3)
    s.set_particles(pos, (np.arange(3000) % 3).astype(np.int32))
    assert s.kernels_per_step() == 5  # no k_zeroth: the births are k_bin's
    run_parity(s, 6, batch=3)
    s.close()
