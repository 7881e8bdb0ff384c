"""The kernel chain of the binned sort (k_bin, k_scan, k_pairs_cells,
k_pairs_big, k_match), on grids of more cells than k_resident takes or with
a panel, GPU against the oracle bit for bit, and its bounded waits.  Bits are
compared, so there is no tolerance."""
import time

import numpy as np
import pytest

from gpusmoldyn_gb300 import _lib as L
from gpusmoldyn_gb300.configs import rng, uniform_positions
from gpusmoldyn_gb300.system import System
from test_gpu_parity import run_parity
from test_gpu_resident import system

pytestmark = pytest.mark.gpu

CELLS = 54  # 157,464 cells of edge 0.25


@pytest.mark.parametrize("births,kernels", [(0.7, 5), (40.0, 5), (499.0, 5), (501.0, 6), (2000.0, 6)])
def test_bins_overflow_beside_births(births, kernels):
    """A cluster overflows its bin while the last CTA of k_bin makes the
    step's births (1,000 by two reactions at most; more are k_zeroth's): the
    step stops whole and is replayed with larger bins."""
    s = system(3000, CELLS, births=births)
    g = rng(17)
    pos = uniform_positions(g, 3000, (0, 0, 0), (0.25 * CELLS,) * 3)
    pos[:400] = uniform_positions(g, 400, (0.3,) * 3, (0.4,) * 3)
    s.set_particles(pos, (np.arange(3000) % 3).astype(np.int32))
    assert s.kernels_per_step() == kernels
    run_parity(s, 6, batch=3)
    s.close()


@pytest.mark.parametrize("sort", ["binned", "compact"])
@pytest.mark.parametrize("n", [2048, 2049, 4097, 65537])
def test_large_cells_without_second_order_reactions(n, sort):
    """Cells cut into units (2,048 records) and joined by one merge pass, or
    by two above 32 units, in a network that has no pairs to find."""
    s = System((-0.75,) * 3, (1.25,) * 3, dt=1e-3, seed=83, normals="table", sort=sort, cell_size=0.5)
    A, B = s.add_species(0.2), s.add_species(0.1)
    s.add_reaction(1, [A], [B], 30.0)
    s.add_reaction(1, [B], [A, A], 20.0)
    if sort == "binned":  # a panel nothing meets, so that the steps are the chain's
        f = s.add_surface()
        s.set_surface_action(f, L.BD_ALL_SPECIES, "both", "transmit")
        s.add_panel(f, "rect", [1.2, -0.75, -0.75, 2.0, 2.0], axis=0)
    s.finalize()
    g = rng(83)
    pos = np.concatenate([uniform_positions(g, n, (-0.15,) * 3, (0.15,) * 3),
                          uniform_positions(g, 300, (0.4,) * 3, (1.25,) * 3)])
    s.set_particles(pos, g.integers(0, 2, len(pos)).astype(np.int32))
    assert s.kernels_per_step() > 1
    run_parity(s, 2)
    s.close()


@pytest.mark.parametrize("n,cells,kernels", [
    (50000, 26, 1),       # 17,576 cells
    (50000, 27, 5),       # 19,683
    (100000, 26, 1),      # the most particles
    (100001, 26, 5),
    (60000, 35, 1),       # 42,875 cells: 1.4 a cell
    (3456, 3, 1),         # 128 a cell
    (3457, 3, 5),         # and one more: large cells are the rule
], ids=lambda v: str(v))
def test_the_line_between_k_resident_and_the_chain(n, cells, kernels):
    s = system(n, cells, kon=0.2)
    assert s.kernels_per_step() == kernels
    run_parity(s, 4, batch=2)
    s.close()


def hidden_panel(s, x, side):
    """A panel that nothing meets: the steps are the chain's, whatever the size."""
    f = s.add_surface()
    s.set_surface_action(f, L.BD_ALL_SPECIES, "both", "transmit")
    s.add_panel(f, "rect", [x, -side, -side, 2 * side, 2 * side], axis=0)


@pytest.mark.parametrize("n,where,kon,steps", [
    (129, (-0.15, 0.15), 0.5, 2),
    (2049, (-0.15, 0.15), 0.02, 2),
    (6000, (0.10, 0.40), 0.02, 3),      # eight large neighbours around a corner
    (65537, (-0.15, 0.15), 0.001, 1),   # 33 units: a second merge pass
], ids=lambda v: str(v))
def test_large_cells_of_the_binned_chain(n, where, kon, steps):
    s = System((-0.75,) * 3, (1.25,) * 3, dt=1e-3, seed=83, normals="table", sort="binned", cell_size=0.5)
    A, B, Cc, X = (s.add_species(d) for d in (0.2, 0.2, 0.1, 0.2))
    s.add_reaction(2, [A, B], [Cc], kon)
    s.add_reaction(1, [Cc], [A, B], 50.0)
    hidden_panel(s, 1.2, 2.0)
    s.finalize()
    g = rng(83)
    pos = np.concatenate([uniform_positions(g, n, (where[0],) * 3, (where[1],) * 3),
                          uniform_positions(g, 300, (0.4,) * 3, (1.25,) * 3)])
    s.set_particles(pos, g.integers(0, 4, len(pos)).astype(np.int32))
    assert s.kernels_per_step() == 6
    _, npairs, _ = run_parity(s, steps)
    assert n < 1000 or npairs > 20
    s.close()


def test_slots_and_pairs_outgrown_on_the_chain():
    s = system(2000, CELLS, births=40.0, capacity=2400)
    assert s.kernels_per_step() == 5
    run_parity(s, 24, batch=12)
    s.close()
    s = System((0, 0, 0), (1.5,) * 3, dt=1e-3, seed=7, normals="table", sort="binned", pair_capacity=64)
    A, B, Cc = s.add_species(1.0), s.add_species(1.0), s.add_species(0.5)
    s.add_reaction(2, [A, B], [Cc], 8.0)
    s.add_reaction(1, [Cc], [A, B], 40.0)
    hidden_panel(s, 1.4, 2.0)
    s.finalize()
    s.set_particles(uniform_positions(rng(7), 6000, (0, 0, 0), (1.5,) * 3), (np.arange(6000) % 3).astype(np.int32))
    assert s.kernels_per_step() == 6
    _, pairs, _ = run_parity(s, 3)
    assert pairs > 8192  # the matching of the whole grid
    s.close()


def times_out(s, withhold):
    L.check(withhold(s.h, 1), "withhold")
    t0 = time.perf_counter()
    s.step(1)
    with pytest.raises(L.BDError) as e:
        s.synchronize()
    assert e.value.code == L.BD_ERR_TIMEOUT
    assert time.perf_counter() - t0 < 30.0
    s.close()


def test_scan_wait_of_the_chain_runs_out():
    """CTA 0 of k_scan never arrives (test switch): the others' waits run out,
    the step ends with BD_ERR_TIMEOUT and the context stays usable."""
    s = system(20000, CELLS)
    assert s.kernels_per_step() == 5
    s.step(2)
    s.synchronize()
    times_out(s, s.lib.bd_debug_withhold_scan)
    s = system(20000, CELLS)
    run_parity(s, 2)
    s.close()


def test_matcher_wait_of_the_chain_runs_out():
    def dense():
        s = System((0, 0, 0), (2.0,) * 3, dt=1e-3, seed=73, normals="table", sort="compact")
        A, B, Cc = s.add_species(1.0), s.add_species(1.0), s.add_species(0.5)
        s.add_reaction(2, [A, B], [Cc], 5.0)
        s.finalize()
        s.set_particles(uniform_positions(rng(73), 4000, (0, 0, 0), (2,) * 3), (np.arange(4000) % 2).astype(np.int32))
        assert s.kernels_per_step() == 6
        return s
    s = dense()
    times_out(s, s.lib.bd_debug_withhold_match)
    s = dense()
    _, pairs, _ = run_parity(s, 1)
    assert pairs > 8192
    s.close()
