"""The cell scan against the oracle bit for bit, over cell counts where its
ranges change: one range, ranges that end in 1 to 3 odd counts, threads' runs
of 16 and of 17 counts, ranges of one full chunk and of more than one, and
more CTAs than ranges.  Bits are compared, so there is no tolerance."""
import numpy as np
import pytest

from gpusmoldyn_gb300.configs import rng, uniform_positions
from gpusmoldyn_gb300.system import System
from test_gpu_parity import run_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,sort", [
    ((1, 1, 1), "compact"),
    ((3, 5, 7), "compact"),         # 105 cells: one range, one odd count
    ((23, 29, 47), "compact"),      # 31,349
    ((74, 75, 73), "binned"),       # 405,150
    ((160, 170, 178), "binned"),    # runs of 16 counts, made 17
    ((193, 197, 196), "binned"),    # 7,452,116: chunks full to 60 counts with 304 CTAs
    ((211, 199, 201), "binned"),    # 8,439,789: two chunks, one odd count
], ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else v)
def test_cell_starts_bit_exact(dims, sort):
    side = 0.25 * np.array(dims)
    s = System((0, 0, 0), tuple(side), dt=1e-3, seed=17, normals="table", sort=sort, cell_size=0.25 * 0.999)
    A, B, Cc = s.add_species(1.0), s.add_species(1.0), s.add_species(0.5)
    s.add_reaction(2, [A, B], [Cc], 0.5)
    s.finalize()
    n = min(60000, 40 * int(np.prod(dims)))
    pos = uniform_positions(rng(17), n, (0, 0, 0), tuple(side))
    s.set_particles(pos, (np.arange(n) % 3).astype(np.int32))
    assert tuple(s.grid()[0]) == dims
    run_parity(s, 2)
    s.close()
