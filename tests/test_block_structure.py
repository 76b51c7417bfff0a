"""The device check for coupled velocity blocks (pm_level_decoupled) on every
kind of nine-block level: one nonzero off-diagonal block, several, all six;
diagonal blocks equal or not.  A level whose A12..A32 hold nonzero values on
active rows is in mode 0 and its mat-vec includes them (1e-12, the FP64
tolerance of the other mat-vec tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OFFDIAG = (1, 2, 3, 5, 6, 7)


@pytest.mark.parametrize("blocks", [(), (1,), (7,), (1, 3), (2, 5, 6), OFFDIAG])
@pytest.mark.parametrize("equal", [True, False])
@pytest.mark.parametrize("levels", [2, 4])
def test_mode_follows_the_values(blocks, equal, levels):
    from to_merge_master_parmoon_gb300 import OseenProblem, PmSolver
    P = OseenProblem(n_levels=levels, nu=1e-2, seed=5)
    rng = np.random.default_rng(1)
    for level in range(levels):
        a = P.arrays(level)
        for k in blocks:
            a["a"][k][:] += 1e-3 * rng.standard_normal(a["a"][k].size)
        if not equal:
            a["a"][4][:] *= 1.5
    S = PmSolver(P.descs)
    want = 0 if blocks else (2 if equal else 1)
    assert [S.level_decoupled(k) for k in range(levels)] == [want] * levels
    x = rng.standard_normal(P.ndof(-1))
    y = P.scipy_matrix() @ x
    assert np.linalg.norm(S.matvec(levels - 1, x) - y) <= 1e-12 * np.linalg.norm(y)
    S.close()
