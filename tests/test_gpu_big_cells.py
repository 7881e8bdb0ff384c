"""Large cells, GPU against the oracle bit for bit.  A cell of more than 128
records is cut into units of 2,048 that CTAs sort one by one, joined 32 at a
time by merge passes, and searched for pairs by warps of 32 seekers: one
record over and under a unit, two units, a full pass of 32 units and one
that needs a second pass, x of both signs in a cell, newborns among the
records, inert species, and large neighbours across faces and corners.
Bits are compared, so there is no tolerance."""
import numpy as np
import pytest

from gpusmoldyn_gb300.configs import rng, uniform_positions
from gpusmoldyn_gb300.system import System
from test_gpu_parity import run_parity

pytestmark = pytest.mark.gpu

LO, HI = -0.75, 1.25  # four cells of 0.5 an axis; the second is [-0.25, 0.25)


def system(n, where, kon, sort, seed):
    s = System((LO,) * 3, (HI,) * 3, dt=1e-3, seed=seed, normals="table", sort=sort, cell_size=0.5)
    A, B, Cc, X = (s.add_species(d) for d in (0.2, 0.2, 0.1, 0.2))
    s.add_reaction(2, [A, B], [Cc], kon)
    s.add_reaction(1, [Cc], [A, B], 50.0)
    s.finalize()
    g = rng(seed)
    cluster = uniform_positions(g, n, (where[0],) * 3, (where[1],) * 3)
    rest = uniform_positions(g, 300, (0.4,) * 3, (HI,) * 3)
    pos = np.concatenate([cluster, rest])
    s.set_particles(pos, g.integers(0, 4, len(pos)).astype(np.int32))
    return s


@pytest.mark.parametrize("sort", ["binned", "compact"])
@pytest.mark.parametrize("n,where,kon,steps", [
    (129, (-0.15, 0.15), 0.5, 2),
    (2048, (-0.15, 0.15), 0.02, 2),
    (2049, (-0.15, 0.15), 0.02, 2),
    (4097, (-0.15, 0.15), 0.01, 2),
    (6000, (0.10, 0.40), 0.02, 3),      # eight large neighbours around a corner
    (65537, (-0.15, 0.15), 0.001, 1),   # 33 units: a second merge pass
], ids=lambda v: str(v))
def test_large_cells_bit_exact(n, where, kon, steps, sort):
    if where[0] < 0:  # the whole cluster is one cell in the first step
        first = system(n, where, kon, sort, seed=83)
        first.step(1)
        first.synchronize()
        assert np.diff(first.cells().astype(np.int64)).max() >= n
        first.close()
    s = system(n, where, kon, sort, seed=83)
    _, npairs, _ = run_parity(s, steps)
    assert n < 1000 or npairs > 20
    s.close()
