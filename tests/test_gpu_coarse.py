"""Poisson solves over the forms of the multigrid hierarchy's coarse end: one
level only, a coarsest level held as a dense map (up to 32 cells an edge),
and a larger one that is swept.

Against the FP64 oracle on the same tables, solved to a relative residual of
1e-10.  The solve here stops at 1e-6; the oracle's psi then differs by the
smooth part of that residual, the same 1e-5 that the mixed-precision tests
derive.
"""
import numpy as np
import pytest

import ggb_cases as K

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64).ravel(), np.asarray(b, np.float64).ravel()
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("N,mixed", [(4, 0), (5, 1), (27, 0), (31, 1), (33, 0), (33, 1), (50, 0), (50, 1), (62, 0),
                                     (66, 0), (66, 1), (100, 0)])
def test_poisson_coarse_forms(gpu, orc64, N, mixed):
    ref = K.poisson(orc64, N, tol=1e-10, tables=K.tables_of(gpu, N))
    got = K.poisson(gpu, N, tol=1e-6, mixed=bool(mixed))
    assert float(got["relres"]) <= 1e-6
    assert rel_l2(got["psi"], ref["psi"]) <= 1e-5
    assert rel_l2(got["vel"], ref["vel"]) <= 5e-5
