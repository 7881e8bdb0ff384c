"""Box-Muller normals: the radius of every uniform against double precision,
within the bound that the documented errors of its two approximations give
(tests/cpp/radius_main.cu), and the same bits whether steps run one by one or
many to a launch, and in k_resident or the kernel chain."""
import os
import subprocess

import numpy as np
import pytest

from gpusmoldyn_gb300 import build
from gpusmoldyn_gb300.configs import rng, uniform_positions
from gpusmoldyn_gb300.system import System
from test_gpu_parity import gpu_records

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_radius_of_every_uniform(tmp_path):
    exe = str(tmp_path / "radius")
    subprocess.run([build.nvcc(), "-O3", "-std=c++17", *build.ARCH, "-I", os.path.join(ROOT, "gpusmoldyn_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "cpp", "radius_main.cu"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr


def diffusing(n):
    s = System((-1, 0, 0), (1, 2, 4), dt=1e-3, seed=97)
    s.add_species(1.0)
    s.add_species(30.0)
    s.finalize()
    s.set_particles(uniform_positions(rng(97), n, (-1, 0, 0), (1, 2, 4)), (np.arange(n) % 2).astype(np.int32))
    return s


@pytest.mark.parametrize("n,steps", [(300, 70), (400003, 21), (400003, 3)])
def test_one_launch_equals_single_steps(n, steps):
    a, b = diffusing(n), diffusing(n)
    a.step(steps)
    for _ in range(steps):
        b.step(1)
    np.testing.assert_array_equal(gpu_records(a), gpu_records(b))
    a.close()
    b.close()


def test_resident_steps_equal_the_chain():
    """The binned sort of a small system (one launch) and the compact sort
    (a chain of kernels)."""
    recs = []
    for sort in ("binned", "compact"):
        s = System((0, 0, 0), (4, 4, 4), dt=1e-3, seed=98, sort=sort)
        A, B, Cc = s.add_species(1.0), s.add_species(1.0), s.add_species(0.5)
        s.add_reaction(2, [A, B], [Cc], 0.5)
        s.add_reaction(1, [Cc], [A, B], 40.0)
        s.finalize()
        s.set_particles(uniform_positions(rng(98), 9000, (0, 0, 0), (4, 4, 4)), (np.arange(9000) % 3).astype(np.int32))
        assert (s.kernels_per_step() == 1) == (sort == "binned")
        s.step(40)
        recs.append(gpu_records(s))
        s.close()
    np.testing.assert_array_equal(*recs)
