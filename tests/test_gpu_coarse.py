"""Poisson solves over the forms of the multigrid hierarchy's coarse end: one
level only (swept), a coarsest level held as a dense map (up to 16 cells an
edge), and a larger one that is swept.

Against the FP64 oracle on the same tables, solved to a relative residual of
1e-10.  The solve here stops at 1e-6; the oracle's psi then differs by the
smooth part of that residual, the same 1e-5 that the mixed-precision tests
derive.
"""
import ctypes as C

import numpy as np
import pytest

import ggb_api as G
import ggb_cases as K

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64).ravel(), np.asarray(b, np.float64).ravel()
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("N,mixed", [(4, 0), (5, 1), (27, 0), (31, 1), (33, 0), (33, 1), (50, 0), (50, 1), (62, 0),
                                     (66, 0), (66, 1), (100, 0), (45, 0), (90, 1), (150, 0), (198, 0)])
def test_poisson_coarse_forms(gpu, orc64, N, mixed):
    ref = K.poisson(orc64, N, tol=1e-10, tables=K.tables_of(gpu, N))
    got = K.poisson(gpu, N, tol=1e-6, mixed=bool(mixed))
    assert float(got["relres"]) <= 1e-6
    assert rel_l2(got["psi"], ref["psi"]) <= 1e-5
    assert rel_l2(got["vel"], ref["vel"]) <= 5e-5


@pytest.mark.parametrize("N,mixed", [(6, 0), (12, 0), (34, 1), (70, 0), (72, 0), (72, 1), (74, 0), (126, 0), (130, 1),
                                     (200, 0), (254, 0), (300, 1), (382, 0), (384, 0), (390, 1), (520, 0)])
def test_poisson_level_forms(gpu, orc64, N, mixed):
    """Both sides of the sizes where a level's operators change form (sparse
    rows, structured interiors, one or several chunks of a block's range, 512
    or 1024 threads), with odd coarse levels among them; bounds as above."""
    ref = K.poisson(orc64, N, tol=1e-10, tables=K.tables_of(gpu, N))
    got = K.poisson(gpu, N, tol=1e-6, mixed=bool(mixed))
    assert float(got["relres"]) <= 1e-6
    assert rel_l2(got["psi"], ref["psi"]) <= 1e-5
    assert rel_l2(got["vel"], ref["vel"]) <= 5e-5


@pytest.mark.parametrize("blocks", [1, 2, 5, 7, 40])
@pytest.mark.parametrize("N,mixed", [(25, 0), (66, 1), (72, 0), (130, 1)])
def test_batched_solve_on_few_blocks(gpu, orc64, N, mixed, blocks):
    """One planet's solve on a share of the blocks (fewer than one per face
    among them: ranges that straddle faces), against the FP64 solve of the
    omega it left; bounds as above."""
    g = gpu.grid(N)
    vel0, band = K.initial_velocity(gpu, g, seed=5)
    fs = G.FluidSim(gpu, g, rotation=2.0, cg_tol=1e-6, mixed=bool(mixed))
    fs.set_state(vel0, band)
    F = (C.POINTER(gpu.T["Fluid"]) * 2)(C.pointer(fs.F))
    b = gpu.lib.ggb_batch_create(1, F, None, None, (C.c_double * 1)(1.0), None)
    gpu.lib.ggb_batch_solve_blocks(b, blocks)
    assert gpu.lib.ggb_batch_step(b, 2) == 0
    got = dict(psi=fs.field("psi").copy(), vel=fs.field("vel", 3).copy())
    omega, relres = fs.field("omega").copy(), fs.F.cg_relres
    gpu.lib.ggb_batch_free(b)
    fs.free()
    g.free()
    ref = K.solve_fp64(orc64, N, K.tables_of(gpu, N), omega)
    assert relres <= 1e-6
    assert rel_l2(got["psi"], ref["psi"]) <= 1e-5
    assert rel_l2(got["vel"], ref["vel"]) <= 5e-5


@pytest.mark.parametrize("N,mixed", [(256, 1), (258, 0), (258, 1), (260, 0), (262, 1)])
def test_poisson_narrow_block_sizes(gpu, orc64, N, mixed):
    """Both sides of the mean cells per block up to which blocks have 384
    threads; bounds as above."""
    ref = K.poisson(orc64, N, tol=1e-10, tables=K.tables_of(gpu, N))
    got = K.poisson(gpu, N, tol=1e-6, mixed=bool(mixed))
    assert float(got["relres"]) <= 1e-6
    assert rel_l2(got["psi"], ref["psi"]) <= 1e-5
    assert rel_l2(got["vel"], ref["vel"]) <= 5e-5


@pytest.mark.parametrize("N,mixed", [(128, 0), (129, 1)])
def test_block_count_does_not_change_the_solve(gpu, N, mixed):
    """Shares of 5 to 12 blocks cut the cells anywhere on the faces: the same
    psi from the same state, to 100 times the FP32 rounding (a sum in FP64 over
    other partial sums moves an FP32 vector by an ulp now and then)."""
    out = []
    for blocks in (5, 6, 11, 12):
        g = gpu.grid(N)
        vel0, band = K.initial_velocity(gpu, g, seed=5)
        fs = G.FluidSim(gpu, g, rotation=2.0, cg_tol=1e-6, mixed=bool(mixed))
        fs.set_state(vel0, band)
        F = (C.POINTER(gpu.T["Fluid"]) * 1)(C.pointer(fs.F))
        b = gpu.lib.ggb_batch_create(1, F, None, None, (C.c_double * 1)(1.0), None)
        gpu.lib.ggb_batch_solve_blocks(b, blocks)
        assert gpu.lib.ggb_batch_step(b, 1) == 0
        out.append(fs.field("psi").copy())
        gpu.lib.ggb_batch_free(b)
        fs.free()
        g.free()
    for psi in out[1:]:
        assert rel_l2(psi, out[0]) <= 1.2e-5
