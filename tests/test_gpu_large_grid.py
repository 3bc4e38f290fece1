"""A fluid without multigrid on a grid beyond the solve's largest edge (1535
cells): it initialises, and what needs no solve works; the solve itself ends the
process with a message.  In a process of its own."""
import subprocess
import sys

import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

RUN = r"""
import ctypes as C, sys
import numpy as np
sys.path.insert(0, {pkg!r})
import ggb_api as G
gpu = G.Api(G.PRODUCT_LIB)
g = gpu.grid(1536)
fs = G.FluidSim(gpu, g, multigrid=0)
# psi = z / 2: a solid-body rotation, |u| = 1 / 2 at the equator
fs.field("psi")[:] = 0.5 * g.arrays()["pos"].reshape(-1, 3)[:, 2]
gpu.lib.fluid_compute_velocity(C.byref(fs.F))
print("speed", fs.max_speed(), flush=True)
fs.solve()
print("solved", flush=True)
"""


def test_fluid_without_multigrid_beyond_the_solve(gpu):
    p = subprocess.run([sys.executable, "-c", RUN.format(pkg=PKG)], capture_output=True, text=True, timeout=300)
    assert p.stdout.startswith("speed "), p.stderr
    assert abs(float(p.stdout.split()[1]) - 0.5) < 1e-4
    assert p.returncode == 1 and "solved" not in p.stdout and "N > 1535" in p.stderr
