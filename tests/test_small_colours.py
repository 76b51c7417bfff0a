"""Sweeps of levels that keep the CSR kernels, on colours too small to fill the
GPU (one CTA per cell: split row groups, shared-out stream, staged LU) and on
colours above those limits, against the oracle's sweeps: FP64 to 1e-9, mixed
to 5e-4, the tolerances of the other Vanka tests.  One cell per colour, uneven
boxes, tetrahedra (48 colours), coupled blocks and distinct diagonal blocks;
the largest hexahedral level has 2,304 cells in a colour."""
import numpy as np
import pytest

from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu

CASES = [
    ("hexa", "coupled", dict(n_levels=2, nx0=1, ny0=1, nz0=1)),
    ("hexa", "coupled", dict(n_levels=3, nx0=3, ny0=1, nz0=2)),
    ("hexa", "diagonal", dict(n_levels=3, nx0=1, ny0=2, nz0=3)),
    ("hexa", "diagonal", dict(n_levels=3, nx0=6, ny0=6, nz0=8)),
    ("hexa", "coupled", dict(n_levels=3, nx0=6, ny0=6, nz0=8)),
    ("tetra", "one", dict(n_levels=2, nx0=1, ny0=1, nz0=1)),
    ("tetra", "one", dict(n_levels=3, nx0=2, ny0=1, nz0=1)),
    ("tetra", "coupled", dict(n_levels=2, nx0=2, ny0=3, nz0=1)),
]


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("element,blocks,mesh", CASES)
def test_sweeps_match_the_oracle(element, blocks, mesh, precision):
    from to_merge_master_parmoon_gb300 import OseenProblem, PmSolver
    box = (0, 0.5 * mesh["nx0"], 0, 0.5 * mesh["ny0"], 0, 0.5 * mesh["nz0"])
    P = OseenProblem(nu=1e-2, seed=2, element=element, box=box, **mesh)
    for level in range(P.n_levels):
        a = P.arrays(level)["a"]
        if blocks == "coupled":
            a[1][:], a[3][:] = -0.05 * a[0], 0.05 * a[0]
        if blocks == "diagonal":
            a[4][:], a[8][:] = 1.5 * a[0], 0.75 * a[0]
    O = Oracle(P)
    S = PmSolver(P.descs, precision=precision)
    level = P.n_levels - 1
    rng = np.random.default_rng(4)
    u, f = 0.1 * rng.standard_normal(P.ndof(level)), rng.standard_normal(P.ndof(level))
    got = S.cell_vanka(level, u, f, 2)
    assert rel(got, O.cell_vanka(level, u, f, 2)) < (1e-9 if precision == "fp64" else 5e-4)
    S.close()
