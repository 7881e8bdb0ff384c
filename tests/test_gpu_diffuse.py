"""Diffusion-only systems, whose steps run many to a launch
(k_diffuse_steps), GPU against the oracle bit for bit: one record, a record
more than a CTA, several launches in a row, steps longer than the box.
Bits are compared, so there is no tolerance."""
import numpy as np
import pytest

from gpusmoldyn_gb300.configs import rng, uniform_positions
from gpusmoldyn_gb300.system import System
from test_gpu_parity import gpu_records, run_parity

pytestmark = pytest.mark.gpu


def system(n, D=(1.0, 0.1, 0.0), side=2.0):
    s = System((-1, 0, 0), (side - 1, side, 2 * side), dt=1e-3, seed=97, normals="table")
    for d in D:
        s.add_species(d)
    s.finalize()
    pos = uniform_positions(rng(97), n, (-1, 0, 0), (side - 1, side, 2 * side))
    s.set_particles(pos, (np.arange(n) % len(D)).astype(np.int32))
    return s


@pytest.mark.parametrize("n,steps,batch,D", [
    (1, 130, 130, (1.0,)),            # three launches
    (257, 66, 33, (1.0, 0.1, 0.0)),
    (100003, 6, 3, (1.0, 0.1, 0.0)),
    (400003, 4, 3, (1.0, 0.1, 0.0)),  # more than a wave of records, few steps
    (400003, 21, 21, (1.0,)),         # and many
    (1000, 4, 2, (5000.0, 1.0)),      # steps that cross the box several times
])
def test_diffusion_steps_in_one_launch_bit_exact(n, steps, batch, D):
    s = system(n, D)
    run_parity(s, steps, batch=batch)
    assert s.step_count() == steps
    s.close()


def test_one_launch_equals_single_steps():
    a, b = system(5000), system(5000)
    a.step(70)
    for _ in range(70):
        b.step(1)
    np.testing.assert_array_equal(gpu_records(a), gpu_records(b))
    assert a.step_count() == b.step_count() == 70
    a.close()
    b.close()
