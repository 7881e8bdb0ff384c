"""Readback of every slot (no slot emptied by the last step, all instances)
against the readback that counts and compacts, and against the slots
themselves.  Bits are compared, so there is no tolerance."""
import numpy as np
import pytest

from gpusmoldyn_gb300 import _lib as L
from gpusmoldyn_gb300.configs import rng, uniform_positions
from gpusmoldyn_gb300.system import System

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kon,steps", [
    (1, 0.0, 3),
    (4097, 0.0, 0),        # straight after the upload
    (50001, 0.0, 2),       # every slot live
    (50001, 30.0, 2),      # slots emptied by the last step
], ids=str)
def test_whole_readback_equals_compacted(n, kon, steps):
    s = System((0, 0, 0), (10, 10, 10), dt=1e-3, seed=5, normals="table")
    A, B, Cc = s.add_species(1.0), s.add_species(1.0), s.add_species(0.5)
    if kon:
        s.add_reaction(2, [A, B], [Cc], kon)
    s.add_reaction(1, [A], [A, B] if n > 1 else [B], 5.0)  # newborns carry a flag in the slot
    s.finalize()
    pos = uniform_positions(rng(5), n, (0, 0, 0), (10, 10, 10))
    s.set_particles(pos, (np.arange(n) % 3).astype(np.int32))
    s.step(steps)
    s.synchronize()
    xyz, w = s.slots()
    live = w != L.DEAD
    assert ((~live).sum() > 0) == (kon > 0)
    whole, one = s.particles4(), s.particles4(instance=0)
    np.testing.assert_array_equal(whole[0].view(np.uint32), one[0].view(np.uint32))
    np.testing.assert_array_equal(whole[1], one[1])
    np.testing.assert_array_equal(whole[0][:, :3], xyz[live])
    s.close()
