"""Handles stepping at the same time on their own streams, more of them than
fit the device together: k_resident on a quarter of the SMs each, the kernel
chain, large cells with and without second-order reactions, diffusion.  Each
ends with the records and events it has alone."""
import numpy as np
import pytest

from gpusmoldyn_gb300.configs import rng, uniform_positions
from gpusmoldyn_gb300.system import System
from test_gpu_parity import gpu_records

pytestmark = pytest.mark.gpu


def make(kind, seed):
    side = 8.0 if kind in ("resident", "diffuse") else 18.0
    n = {"resident": 20003, "chain": 120001, "crowded": 20003, "crowded_first_order": 20003, "diffuse": 50001}[kind]
    s = System((0, 0, 0), (side,) * 3, dt=1e-3, seed=seed, normals="table",
               sort="compact" if kind.startswith("crowded") else "auto")
    A, B, Cc = s.add_species(1.0), s.add_species(1.0), s.add_species(0.5)
    if kind != "diffuse":
        s.add_reaction(1, [Cc], [A, B], 20.0)
        if kind != "crowded_first_order":
            s.add_reaction(2, [A, B], [Cc], 0.02)
    s.finalize()
    pos = uniform_positions(rng(seed), n, (0, 0, 0), (side,) * 3)
    if kind.startswith("crowded"):
        pos[:6000] = uniform_positions(rng(seed + 1), 6000, (0.1,) * 3, (0.25,) * 3)
    s.set_particles(pos, (np.arange(n) % 3).astype(np.int32))
    assert s.kernels_per_step() == (1 if kind in ("resident", "diffuse") else 5 if kind == "chain" else 6)
    return s


def test_many_handles_step_together_as_alone():
    kinds = (["resident"] * 6 + ["chain", "crowded", "crowded_first_order", "diffuse"]) * 2
    alone = []
    for k, kind in enumerate(kinds):
        s = make(kind, 300 + k)
        s.step(30)
        alone.append((gpu_records(s), s.event_counts()))
        s.close()
    handles = [make(kind, 300 + k) for k, kind in enumerate(kinds)]
    for burst in (1, 1, 1, 7, 20):
        for s in handles:
            s.step(burst)
    for s, (records, events) in zip(handles, alone):
        np.testing.assert_array_equal(gpu_records(s), records)
        np.testing.assert_array_equal(s.event_counts(), events)
        s.close()
