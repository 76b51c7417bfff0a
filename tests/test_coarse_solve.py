"""The coarse direct solve over the sizes of its kernels: one-block LU, panels
shared out over a cluster, inverse by one warp per column (up to 1,152
unknowns) and by one CTA per column above, GEMV by one warp per row.  The LU
solve of pm_solve_exact and the inverse used in the V-cycle against a dense
FP64 solve of the pinned system (relative 1e-9; condition up to 1e5)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1, 1, 1), (2, 1, 1), (2, 2, 2), (3, 2, 2), (3, 3, 3), (4, 3, 3)])
def test_lu_and_inverse(n):
    from to_merge_master_parmoon_gb300 import OseenProblem, PmSolver
    P = OseenProblem(n_levels=1, nu=1e-2, seed=1, nx0=n[0], ny0=n[1], nz0=n[2])
    S = PmSolver(P.descs, precision="fp64")
    nu3, N = 3 * P.desc(0).n_udof, P.ndof(0)
    K = P.scipy_matrix(0).toarray()
    K[nu3] = 0.0
    K[nu3, nu3] = 1.0
    b = np.random.default_rng(0).standard_normal(N)
    c = b.copy()
    c[nu3] = 0.0
    want = np.linalg.solve(K, c)
    for got in (S.solve_exact(b), S.vcycle(b)):
        assert np.linalg.norm(got - want) <= 1e-9 * np.linalg.norm(want)
    S.close()
