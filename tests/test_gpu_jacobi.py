"""Solves without multigrid (the Jacobi preconditioner): a fixed number of CG
iterations from psi = 0 against the FP64 restatement on the same tables, at grid
sizes on both sides of where a block's cells fill a pass of its threads or four
passes, of the block sizes (384, 512 and 1024 threads), and with fewer cells than
blocks.

CG iterates agree while rounding has not been amplified: every FP32 vector is
rounded once an iteration (6e-8), the residual's error enters psi through alpha
(a few, here) and 20 iterations add up; 1e-5 leaves a factor of two to eight.
The smallest grids iterate 2 N times: with 96 cells CG is at FP64 rounding after 14
iterations, where no FP32 solve follows it."""
import ctypes as C

import numpy as np
import pytest

import ggb_api as G
import ggb_cases as K

pytestmark = pytest.mark.gpu


def solve(api, N, tables=None, maxit=20):
    g = api.grid(N)
    if tables is not None:
        K.load_tables(api, g, tables)
    fs = G.FluidSim(api, g, cg_tol=1e-12, cg_maxit=maxit, multigrid=0)
    fs.field("omega")[:] = K.lap_exact(g.arrays()["pos"].astype(np.float64)).astype(api.np_real)
    api.lib.fluid_remove_mean(C.byref(g.cs), fs.F.omega)
    it = fs.solve()
    psi, relres = fs.field("psi").astype(np.float64).copy(), fs.F.cg_relres
    fs.free()
    g.free()
    return it, psi, relres


@pytest.mark.parametrize("N", [4, 5, 12, 96, 98, 112, 113, 192, 194, 258, 260, 478, 480])
def test_jacobi_iterations(gpu, orc64, N):
    maxit = min(20, 2 * N)
    ref_it, ref, ref_relres = solve(orc64, N, K.tables_of(gpu, N), maxit)
    it, psi, relres = solve(gpu, N, maxit=maxit)
    assert it == ref_it
    assert np.linalg.norm(psi - ref) <= 1e-5 * np.linalg.norm(ref)
    assert abs(relres - ref_relres) <= 1e-4 * ref_relres + 1e-9
