"""Small binned systems, whose steps run many to a launch (k_resident), GPU
against the oracle bit for bit: cell counts on both sides of the limits
where every CTA keeps all cell starts and where the kernel chain takes
over, systems of a few records, launches in a row, steps with and without
candidate pairs, zeroth-order births with one and two products, a step
that fails in the middle of a launch and is replayed, and a matching that
takes the whole grid.  Bits are compared, so there is no tolerance."""
import numpy as np
import pytest

from gpusmoldyn_gb300.configs import rng, uniform_positions
from gpusmoldyn_gb300.system import System
from test_gpu_parity import run_parity

pytestmark = pytest.mark.gpu


def system(n, cells, kon=0.5, births=0.0, seed=91, **kw):
    """Particles in a cube of cells^3 cells of edge 0.25."""
    side = 0.25 * cells
    s = System((0, 0, 0), (side,) * 3, dt=1e-3, seed=seed, normals="table", sort="binned", cell_size=0.25 * 0.999, **kw)
    A, B, Cc = s.add_species(1.0), s.add_species(1.0), s.add_species(0.5)
    s.add_reaction(2, [A, B], [Cc], kon)
    s.add_reaction(1, [Cc], [A, B], 40.0)
    s.add_reaction(2, [A, A], [B], 0.1)
    if births:  # mean births per step, each
        s.add_reaction(0, [], [A], births / (1e-3 * side ** 3))
        s.add_reaction(0, [], [A, Cc], births / (1e-3 * side ** 3))
    s.finalize()
    pos = uniform_positions(rng(seed), n, (0, 0, 0), (side,) * 3)
    s.set_particles(pos, (np.arange(n) % 3).astype(np.int32))
    return s


@pytest.mark.parametrize("n,cells,steps,batch", [
    (1, 4, 5, 5),
    (7, 5, 130, 130),         # three launches in a row, mostly without candidates
    (3000, 7, 70, 35),
    (40000, 31, 6, 3),        # 29,791 cells: starts in shared memory
    (40000, 33, 6, 3),        # 35,937: a range per CTA
    (200000, 53, 4, 2),       # 148,877: the most cells in one launch
    (200000, 54, 4, 2),       # 157,464: the kernel chain
    (200000, 74, 4, 2),       # 405,224
], ids=lambda v: str(v))
def test_steps_in_one_launch_bit_exact(n, cells, steps, batch):
    s = system(n, cells, births=3.0 if n > 1 else 0.0)
    assert int(np.prod(s.grid()[0].astype(np.int64))) == cells ** 3
    resident = cells < 54
    assert s.kernels_per_step() == 1 if resident else s.kernels_per_step() > 1
    run_parity(s, steps, batch=batch)
    s.close()


def test_failed_step_in_a_launch_is_replayed():
    """Births outgrow the slots in the middle of a launch, and a cluster its
    bins at the first step."""
    s = system(2000, 6, births=40.0, capacity=2400)
    run_parity(s, 48, batch=24)
    s.close()
    s = system(2000, 6)
    g = rng(5)
    pos = uniform_positions(g, 3000, (0, 0, 0), (1.5,) * 3)
    pos[:400] = uniform_positions(g, 400, (0.3,) * 3, (0.4,) * 3)
    s.set_particles(pos, (np.arange(3000) % 3).astype(np.int32))
    run_parity(s, 20, batch=10)
    s.close()


def test_whole_grid_matching_in_a_launch():
    s = system(6000, 6, kon=8.0)
    _, pairs, _ = run_parity(s, 3, batch=1)
    assert pairs > 8192
    s.close()
    s = system(6000, 6, kon=8.0)
    run_parity(s, 6, batch=6)
    s.close()


def test_ensemble_in_one_launch():
    """Instances of an ensemble, many steps to a launch, equal each alone."""
    inst = [dict(box_lo=(0, 0, 0), box_hi=(1.0 + 0.5 * k,) * 3, seed=7 + k, d_scale=1.0 + k, k2_scale=1.0)
            for k in range(3)]

    def make(which):
        s = System(dt=1e-3, instances=which, normals="table", sort="binned")
        A, B, Cc = s.add_species(1.0), s.add_species(1.0), s.add_species(0.5)
        s.add_reaction(2, [A, B], [Cc], 0.5)
        s.add_reaction(1, [Cc], [A, B], 40.0)
        s.add_reaction(0, [], [A], 500.0)
        s.finalize()
        pos = [uniform_positions(rng(d["seed"]), 500 * (1 + i), d["box_lo"], d["box_hi"]) for i, d in enumerate(which)]
        cnt = [len(q) for q in pos]
        s.set_ensemble_particles(np.concatenate(pos), np.arange(sum(cnt)) % 3, cnt)
        return s, cnt
    s, cnt = make(inst)
    s.step(20)
    together = [s.particles(k) for k in range(3)]
    s.close()
    for k in range(3):
        one = System(dt=1e-3, instances=[inst[k]], normals="table", sort="compact")
        A, B, Cc = one.add_species(1.0), one.add_species(1.0), one.add_species(0.5)
        one.add_reaction(2, [A, B], [Cc], 0.5)
        one.add_reaction(1, [Cc], [A, B], 40.0)
        one.add_reaction(0, [], [A], 500.0)
        one.finalize()
        pos = uniform_positions(rng(inst[k]["seed"]), cnt[k], inst[k]["box_lo"], inst[k]["box_hi"])
        first = sum(cnt[:k])
        one.set_particles(pos, (np.arange(first, first + cnt[k]) % 3).astype(np.int32))
        one.step(20)
        p, sp = one.particles()
        one.close()
        np.testing.assert_array_equal(p.view(np.uint32), together[k][0].view(np.uint32))
        np.testing.assert_array_equal(sp, together[k][1])
