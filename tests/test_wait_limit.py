"""A wait for a bulk copy that runs out (wait_limit = 1: the copies just issued
cannot have landed) in every sweep kernel that is fed by such copies: packed
sweeps in FP32 and FP64 (one CTA per cell, and CTAs that walk several cells,
with one stage and with two), and the staged LU apply on hexahedra (the 9.6 KB of a
tetrahedron have landed before the kernel polls).  The kernels stop writing, wait for the copies in flight and
return, the call reports PM_TIMEOUT, and a handle with the default limit then
sweeps as one did before."""
import numpy as np
import pytest

PM_TIMEOUT = 4

pytestmark = pytest.mark.gpu

CUBE = dict(n_levels=3)
WIDE = dict(n_levels=3, nx0=4, ny0=4, nz0=5)  # 640 cells in a colour
CASES = [
    ("mixed", {}, CUBE), ("fp64", {}, CUBE), ("mixed", {}, WIDE), ("fp64", {}, WIDE),
    ("fp64", {}, dict(n_levels=4)),
    ("mixed", dict(decouple=0), CUBE), ("fp64", dict(decouple=0), CUBE),
]


@pytest.mark.parametrize("precision,options,mesh", CASES)
def test_wait_that_runs_out(precision, options, mesh):
    from to_merge_master_parmoon_gb300 import OseenProblem, PmError, PmSolver
    P = OseenProblem(nu=1e-2, seed=3, **mesh)
    level = P.n_levels - 1
    rng = np.random.default_rng(1)
    u, f = 0.1 * rng.standard_normal(P.ndof(level)), rng.standard_normal(P.ndof(level))

    def sweep(**extra):
        S = PmSolver(P.descs, precision=precision, **options, **extra)
        try:
            return S.cell_vanka(level, u, f, 2)
        finally:
            S.close()

    want = sweep()
    with pytest.raises(PmError) as e:
        sweep(wait_limit=1)
    assert e.value.status == PM_TIMEOUT
    assert np.array_equal(sweep(), want)
