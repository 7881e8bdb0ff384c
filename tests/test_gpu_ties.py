"""Large cells whose molecules share x bits, GPU against the oracle bit for
bit: a plane, a line, a point (immobile species), stretches of equal x around
the length from which a unit is sorted by all four words, identical records,
and a mixture with mobile ones.  Bits are compared, so there is no
tolerance."""
import numpy as np
import pytest

from gpusmoldyn_gb300.configs import rng, uniform_positions
from gpusmoldyn_gb300.system import System
from test_gpu_parity import run_parity

pytestmark = pytest.mark.gpu


def place(mode, n, g):
    pos = uniform_positions(g, n, (-0.4,) * 3, (0.4,) * 3)
    if mode == "plane":
        pos[:, 0] = -0.125
    elif mode == "line":
        pos[:, :2] = 0.25
    elif mode == "point":
        pos[:] = 0.125
    elif mode == "half":
        pos[: n // 2, 0] = 0.0
        pos[n // 2:, 0] *= -1.0
    else:  # stretches of so many records with one x
        k = int(mode)
        pos[:, 0] = np.repeat(pos[: n // k + 1, 0], k)[:n]
    return pos


@pytest.mark.parametrize("sort", ["binned", "compact"])
@pytest.mark.parametrize("mode,n,mobile", [
    ("plane", 129, 0.0), ("plane", 2048, 0.0), ("plane", 5000, 0.0), ("line", 3000, 0.0), ("point", 2049, 0.0),
    ("half", 4097, 0.0), ("half", 3000, 0.3), ("7", 2100, 0.0), ("8", 2048, 0.0), ("9", 2048, 0.0), ("10", 4000, 0.5),
], ids=lambda v: str(v))
def test_equal_x_bits(mode, n, mobile, sort):
    s = System((-0.5,) * 3, (1.5,) * 3, dt=1e-3, seed=89, normals="table", sort=sort, cell_size=1.0)
    A, B, M = s.add_species(0.0), s.add_species(0.0), s.add_species(0.05)
    s.add_reaction(2, [A, M], [B, M], 0.001)
    s.add_reaction(1, [A], [B], 5.0)
    s.finalize()
    g = rng(89)
    sp = g.integers(0, 2, n).astype(np.int32)
    sp[g.random(n) < mobile] = M
    s.set_particles(place(mode, n, g), sp)
    run_parity(s, 3)
    s.close()
