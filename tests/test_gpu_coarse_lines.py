"""Poisson solves on both sides of the lines between the forms of a hierarchy's
coarse end.  A single level (odd N) is swept by one block in shared memory up to
1536 cells (N = 15), with a thread for every cell up to 512 (N = 9), and by the
whole grid above; a coarsest level of a deeper hierarchy is a dense map up to 1536
cells (N = 30 ends at 15) and swept above (N = 34 ends at 17).

Against the FP64 oracle on the same tables, solved to a relative residual of
1e-10.  The solve here stops at 1e-6; psi then differs by the smooth part of that
residual, the 1e-5 of the mixed-precision tests."""
import numpy as np
import pytest

import ggb_cases as K

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64).ravel(), np.asarray(b, np.float64).ravel()
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("N", [7, 9, 11, 13, 15, 17, 30, 34])
def test_poisson_coarse_lines(gpu, orc64, N, mixed):
    ref = K.poisson(orc64, N, tol=1e-10, tables=K.tables_of(gpu, N))
    got = K.poisson(gpu, N, tol=1e-6, mixed=bool(mixed))
    assert float(got["relres"]) <= 1e-6
    assert rel_l2(got["psi"], ref["psi"]) <= 1e-5
    assert rel_l2(got["vel"], ref["vel"]) <= 5e-5
