"""Levels without Dirichlet nodes (the Dirichlet rows are identity rows of the
matrix and count as active): nothing is launched between the conversion of the
right-hand side and the first colour of a sweep.  The default kernels against
named ones (FP32 bit for bit, FP64 to 1e-12), every call with another
right-hand side."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("decouple", [0, 1])
@pytest.mark.parametrize("element", ["hexa", "tetra"])
def test_every_node_active(element, decouple, precision):
    from to_merge_master_parmoon_gb300 import OseenProblem, PmSolver
    from to_merge_master_parmoon_gb300._lib import PmLevelDesc
    P = OseenProblem(n_levels=3, nu=1e-2, seed=3, element=element)
    descs = (PmLevelDesc * P.n_levels)()
    for level in range(P.n_levels):
        C.pointer(descs[level])[0] = P.desc(level)
        d, arrays = descs[level], P.arrays(level)
        for k in (1, 2, 3, 5, 6, 7):  # zeroed by the upload on Dirichlet rows
            arrays["a"][k][arrays["a_rowptr"][arrays["n_active"]]:] = 0.0
        d.n_active = d.hanging_bound = d.n_udof
        d.n_dirichlet = 0
    family = 2 if element == "hexa" and precision == "mixed" and not decouple else 1
    A = PmSolver(descs, precision=precision, decouple=decouple)
    B = PmSolver(descs, precision=precision, decouple=decouple, residual_variant=family,
                 apply_variant=2 if precision == "mixed" else 1)
    rng = np.random.default_rng(5)
    for level in (1, 2):
        u = 0.1 * rng.standard_normal(P.ndof(level))
        for _ in range(6):
            f = rng.standard_normal(P.ndof(level))
            a, b = A.cell_vanka(level, u, f, 1), B.cell_vanka(level, u, f, 1)
            if precision == "mixed":
                assert np.array_equal(a, b)
            else:
                assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)
    A.close()
    B.close()
