"""The panel grid: fine while a step stays within a few boxes, coarse when
steps are long (on the CPU, tests/cpp/panel_grid_main.cpp), and scenes whose
steps cross many boxes, GPU against the oracle bit for bit."""
import os
import subprocess

import numpy as np
import pytest

from gpusmoldyn_gb300.configs import rng, uniform_positions
from gpusmoldyn_gb300.system import System
from surface_cases import mixed_scene

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_boxes_follow_the_step(tmp_path):
    exe = str(tmp_path / "panel_grid")
    csrc = os.path.join(ROOT, "gpusmoldyn_gb300", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", csrc, "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "panel_grid_main.cpp"), os.path.join(csrc, "bd_surface.cpp"),
                    "-lpthread", "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout + out.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("sort", ["binned", "compact"])
@pytest.mark.parametrize("dt", [1e-4, 0.02, 0.5])  # rms steps of 0.002 to 0.24 of the box
def test_long_and_short_steps_bit_exact(dt, sort):
    from test_gpu_parity import run_parity
    s = System((0, 0, 0), (6, 6, 6), dt=dt, seed=31, normals="table", sort=sort)
    species = [s.add_species(d) for d in (1.0, 0.5, 2.0, 1.5)]
    s.add_reaction(1, [species[2]], [species[0], species[1]], 0.2 / dt)
    mixed_scene(s, *species)
    s.finalize()
    s.set_particles(uniform_positions(rng(31), 4000, (0, 0, 0), (6, 6, 6)), (np.arange(4000) % 4).astype(np.int32))
    run_parity(s, 4)
    s.close()
