"""A solve that turns NaN part way ends there, as upstream's loop does
(src/fluid.c:290-358: it goes on while rr > tol2, which a NaN is not).

psi starts as +-1e38: its differences are finite in FP32, so b.b is finite and
the first r.r is not NaN in either precision, but K psi overflows an FP32
residual, and r.r is NaN after the first iteration.
The iteration count has to be the restatement's."""
import ctypes as C
import math

import numpy as np
import pytest

import ggb_api as G
import ggb_cases as K

pytestmark = pytest.mark.gpu

SOLVE_NONFINITE, SOLVE_MAXIT = 2, 8


def overflowing_state(api, g, fs):
    fs.field("omega")[:] = K.lap_exact(g.arrays()["pos"].astype(np.float64)).astype(np.float32)
    fs.field("psi")[:] = np.where(np.arange(g.n) % 2, 1e38, -1e38).astype(np.float32)


def solve(api, N, multigrid, mixed=False, maxit=60):
    g = api.grid(N)
    fs = G.FluidSim(api, g, cg_tol=1e-6, cg_maxit=maxit, multigrid=multigrid, mixed=mixed)
    overflowing_state(api, g, fs)
    it, relres = fs.solve(), fs.F.cg_relres
    flags = api.lib.ggb_solve_flags(C.byref(fs.F)) if api.has("ggb_solve_flags") else None
    fs.free()
    g.free()
    return it, relres, flags


# one level swept by a block and by the grid, a dense map, swept coarsest levels, no multigrid
@pytest.mark.parametrize("N,multigrid,mixed", [(5, 1, 0), (17, 1, 0), (17, 1, 1), (16, 1, 0), (64, 1, 0), (64, 1, 1),
                                               (66, 1, 0), (16, 0, 0), (33, 0, 0)])
def test_nan_part_way_ends_the_solve(gpu, orc32, N, multigrid, mixed):
    ref_it, ref_relres, _ = solve(orc32, N, multigrid)
    assert ref_it == 1 and math.isnan(ref_relres)
    it, relres, flags = solve(gpu, N, multigrid, bool(mixed))
    assert it == ref_it and math.isnan(relres)
    assert flags & SOLVE_NONFINITE and not flags & SOLVE_MAXIT


def test_nan_planet_does_not_hold_up_a_batch(gpu):
    """The same state in one planet of a batch: it stops as it does alone, and
    the planet beside it converges."""
    g = gpu.grid(32)
    fluids = [G.FluidSim(gpu, g, cg_tol=1e-6, cg_maxit=60) for _ in range(2)]
    for fs in fluids:
        fs.set_state(K.initial_velocity(gpu, g, seed=5)[0])
    fluids[0].field("psi")[:] = np.where(np.arange(g.n) % 2, 1e38, -1e38).astype(np.float32)
    F = (C.POINTER(gpu.T["Fluid"]) * 2)(*[C.pointer(fs.F) for fs in fluids])
    b = gpu.lib.ggb_batch_create(2, F, None, None, (C.c_double * 2)(1.0, 1.0), None)
    assert gpu.lib.ggb_batch_step(b, 1) == 0
    gpu.lib.ggb_batch_free(b)
    bad, good = fluids
    assert bad.F.cg_iters == 1 and math.isnan(bad.F.cg_relres)
    assert gpu.lib.ggb_solve_flags(C.byref(bad.F)) & SOLVE_NONFINITE
    assert gpu.lib.ggb_solve_flags(C.byref(good.F)) == 0 and good.F.cg_relres <= 1e-6
    for fs in fluids:
        fs.free()
    g.free()
