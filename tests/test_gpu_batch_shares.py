"""Batched solves on shares of a few to many blocks: both forms of the dense
coarse map's product (two warps a row up to two rounds, whole rows beyond), maps
with and without padding columns, and mixtures of sizes.  Against the FP64 solve
of the omega that the step left; the bounds are those of the other batched
solves (the solve stops at 1e-6, psi then differs by the smooth part of that
residual)."""
import ctypes as C

import numpy as np
import pytest

import ggb_api as G
import ggb_cases as K

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64).ravel(), np.asarray(b, np.float64).ravel()
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def step_batch(gpu, sizes, mixed, blocks=0):
    """One batched step of planets of these edges; (omega, psi, velocity, relres) of each."""
    grids = {N: gpu.grid(N) for N in set(sizes)}
    fluids = []
    for k, N in enumerate(sizes):
        fs = G.FluidSim(gpu, grids[N], rotation=2.0, cg_tol=1e-6, mixed=bool(mixed))
        fs.set_state(*K.initial_velocity(gpu, grids[N], seed=5 + k % 3))
        fluids.append(fs)
    n = len(fluids)
    F = (C.POINTER(gpu.T["Fluid"]) * n)(*[C.pointer(fs.F) for fs in fluids])
    b = gpu.lib.ggb_batch_create(n, F, None, None, (C.c_double * n)(*[1.0] * n), None)
    gpu.lib.ggb_batch_solve_blocks(b, blocks)
    assert gpu.lib.ggb_batch_step(b, 1) == 0
    out = [(fs.field("omega").copy(), fs.field("psi").copy(), fs.field("vel", 3).copy(), fs.F.cg_relres)
           for fs in fluids]
    gpu.lib.ggb_batch_free(b)
    for fs in fluids:
        fs.free()
    for g in grids.values():
        g.free()
    return out


def check(gpu, orc64, N, state):
    omega, psi, vel, relres = state
    ref = K.solve_fp64(orc64, N, K.tables_of(gpu, N), omega)
    assert relres <= 1e-6
    assert rel_l2(psi, ref["psi"]) <= 1e-5
    assert rel_l2(vel, ref["vel"]) <= 5e-5


# with 512 threads (16 warps) 30 and 95 blocks are the last that take whole rows of the 486- and 1536-row maps
@pytest.mark.parametrize("N,mixed", [(36, 0), (64, 0), (64, 1)])
@pytest.mark.parametrize("blocks", [1, 3, 13, 30, 31, 40, 41, 95, 96, 127, 128])
def test_dense_map_on_shares(gpu, orc64, N, mixed, blocks):
    check(gpu, orc64, N, step_batch(gpu, [N], mixed, blocks)[0])


# launches with 384, 512 and 1024 threads a block, dense maps, swept levels and single levels side by side
@pytest.mark.parametrize("sizes,mixed", [([64, 64], 0), ([9, 32], 0), ([17, 64, 25], 0), ([66, 32, 64, 50], 1),
                                         ([32] * 24, 0), ([64] * 14, 1), ([25] * 12, 0)])
def test_mixed_batches(gpu, orc64, sizes, mixed):
    out = step_batch(gpu, sizes, mixed)
    done = set()
    for N, state in zip(sizes, out):
        assert state[3] <= 1e-6
        if N not in done:  # one planet of each size against the oracle
            check(gpu, orc64, N, state)
        done.add(N)
