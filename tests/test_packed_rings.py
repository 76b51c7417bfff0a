"""Packed sweeps whose CTAs walk many cells: the stages of packed rows and
factors, the ring of patch lists, the gathered patches and the barriers between
row and solver warps are used over and over, with remainders (colours that are
no multiple of the number of CTAs).  Finest levels of 600 and 640 cells in a
colour (FP64 has two stages up to 608 on 152 SMs, one above), 3,840 and 4,096.
As in the tests of the small levels: against residual_variant=1, FP32 bit for
bit, FP64 to 1e-12 (sums in another order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MESHES = {
    "600": dict(n_levels=3, nx0=3, ny0=5, nz0=5),
    "640": dict(n_levels=3, nx0=4, ny0=4, nz0=5),
    "3840": dict(n_levels=4, nx0=5, ny0=3, nz0=4),
    "4096": dict(n_levels=5, nx0=2, ny0=2, nz0=2),
}


@pytest.fixture(scope="module", params=list(MESHES))
def finest(request):
    from to_merge_master_parmoon_gb300 import OseenProblem
    kw = MESHES[request.param]
    box = (0, 0.5 * kw["nx0"], 0, 0.5 * kw["ny0"], 0, 0.5 * kw["nz0"])
    P = OseenProblem(nu=1e-2, seed=3, box=box, **kw)
    assert P.desc(P.n_levels - 1).n_cells == 8 * int(request.param)
    return P


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_equal_to_the_csr_kernels(finest, precision):
    from to_merge_master_parmoon_gb300 import PmSolver
    level = finest.n_levels - 1
    A = PmSolver(finest.descs, precision=precision, restart=2)
    B = PmSolver(finest.descs, precision=precision, restart=2, residual_variant=1)
    rng = np.random.default_rng(0)
    u, f = 0.1 * rng.standard_normal(finest.ndof(level)), rng.standard_normal(finest.ndof(level))
    for sweeps in (1, 2, 3):
        a, b = A.cell_vanka(level, u, f, sweeps), B.cell_vanka(level, u, f, sweeps)
        if precision == "mixed":
            assert np.array_equal(a, b)
        else:
            assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)
    assert A.packed_bytes > 0 and B.packed_bytes == 0
    A.close()
    B.close()
