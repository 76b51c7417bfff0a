"""Sweeps and V-cycles between an assembly and the refactorisation that
follows it: the residual is formed from the present A, B and BT (also B with
another scale, as after a changed time step), the local solves use the factors
made last.  The default kernels against residual_variant=1 (CSR rows): FP32
bit for bit; FP64, whose sums run in another order, to 1e-12 for two sweeps and
1e-10 for a V-cycle (the coarse inverse, of condition up to 1e5, carries the
2e-16 of the sums)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("one_block", [True, False])
def test_present_values_before_a_refactorisation(precision, one_block):
    from to_merge_master_parmoon_gb300 import OseenProblem, PmSolver
    P = OseenProblem(n_levels=3, nu=1e-2, seed=3)
    descs = P.descs_one_block() if one_block else P.descs
    A = PmSolver(descs, precision=precision)
    B = PmSolver(descs, precision=precision, residual_variant=1)
    rng = np.random.default_rng(2)
    u, f = 0.1 * rng.standard_normal(P.ndof(2)), rng.standard_normal(P.ndof(2))

    def agree():
        for a, b, tol in ((A.cell_vanka(2, u, f, 2), B.cell_vanka(2, u, f, 2), 1e-12),
                          (A.vcycle(f), B.vcycle(f), 1e-10)):
            if precision == "mixed":
                assert np.array_equal(a, b)
            else:
                assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)

    # scales of B and BT; the second returns to the values of the factors
    for b_scale, refactor in ((0.5, False), (1.0, False), (0.25, True), (0.25, False), (2.0, False)):
        for S in (A, B):
            for k in range(3):
                S.assemble_system_level(k, P.cell_sizes(k), P.convection_nodal(k), P.nu, 1.0, 1.0,
                                        b_scale=b_scale, bt_scale=b_scale)
        agree()
        if refactor:
            for S in (A, B):
                S.refactor()
            agree()
    A.close()
    B.close()
