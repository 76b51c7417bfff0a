"""Which sweep kernels run.  The default takes one CTA per cell on colours too
small to fill the GPU, with the sums of the kernels for large colours in the
same order; residual_variant / apply_variant 1 and 2 run the kernel they name
on every colour.  Default against named kernels below the limits (8, 64 and 512
cells in a colour; FP32 bit for bit, FP64 to 1e-12), the names of the kernels
as the profiler sees them, and tetrahedra above the limits (4,096 cells in a
colour) against the oracle with the tolerances of the other sweep tests."""
import numpy as np
import pytest

from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu

# what keeps the level on CSR rows, residual_variant of its default family
LEVELS = [("hexa", "coupled", "mixed", 2), ("hexa", "coupled", "fp64", 1),
          ("hexa", "diagonal", "mixed", 1), ("hexa", "diagonal", "fp64", 1),
          ("tetra", "one", "mixed", 1), ("tetra", "one", "fp64", 1)]


def problem(element, blocks, levels):
    from to_merge_master_parmoon_gb300 import OseenProblem
    P = OseenProblem(n_levels=levels, nu=1e-2, seed=2, element=element)
    for level in range(levels):
        a = P.arrays(level)["a"]
        if blocks == "coupled":
            a[1][:], a[3][:] = -0.05 * a[0], 0.05 * a[0]
        if blocks == "diagonal":
            a[4][:], a[8][:] = 1.5 * a[0], 0.75 * a[0]
    return P


def vectors(P, level):
    rng = np.random.default_rng(4)
    return 0.1 * rng.standard_normal(P.ndof(level)), rng.standard_normal(P.ndof(level))


@pytest.mark.parametrize("element,blocks,precision,family", LEVELS)
def test_small_colours_equal_the_named_kernels(element, blocks, precision, family):
    from to_merge_master_parmoon_gb300 import PmSolver
    P = problem(element, blocks, 4 if element == "hexa" else 3)
    A = PmSolver(P.descs, precision=precision)
    # one cell per warp in FP32, pairs in FP64: the default apply of each
    B = PmSolver(P.descs, precision=precision, residual_variant=family,
                 apply_variant=2 if precision == "mixed" else 1)
    for level in range(1, P.n_levels):
        u, f = vectors(P, level)
        a, b = A.cell_vanka(level, u, f, 2), B.cell_vanka(level, u, f, 2)
        if precision == "mixed":
            assert np.array_equal(a, b)
        else:
            assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)
    A.close()
    B.close()


@pytest.mark.parametrize("element,precision,residual,apply,names", [
    ("hexa", "mixed", 1, 2, ("k_vanka_residual_rows<", "k_vanka_apply<")),
    ("hexa", "mixed", 2, 2, ("k_vanka_residual<", "k_vanka_apply<")),
    ("hexa", "fp64", 1, 1, ("k_vanka_residual_rows<", "k_vanka_apply2<")),
    ("hexa", "fp64", 2, 2, ("k_vanka_residual<", "k_vanka_apply<")),
    ("tetra", "mixed", 1, 2, ("k_vanka_residual_rows<", "k_vanka_apply<")),
    ("tetra", "fp64", 1, 1, ("k_vanka_residual_rows<", "k_vanka_apply2<")),
    ("hexa", "mixed", 0, 0, ("k_vanka_residual_wide<", "k_vanka_apply_staged<")),
    ("tetra", "fp64", 0, 0, ("k_vanka_residual_split<", "k_vanka_apply_staged<")),
])
def test_named_kernels_run(element, precision, residual, apply, names):
    import torch
    from torch.profiler import ProfilerActivity, profile
    from to_merge_master_parmoon_gb300 import PmSolver
    P = problem(element, "coupled" if element == "hexa" else "one", 2)
    S = PmSolver(P.descs, precision=precision, residual_variant=residual, apply_variant=apply)
    u, f = vectors(P, 1)
    for _ in range(2):  # the first profile of a process may miss its kernels
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
            S.cell_vanka(1, u, f, 1)
            torch.cuda.synchronize()
    S.close()
    ran = {e.name.split("k_vanka_", 1)[1].split("<")[0] for e in prof.events()
           if "k_vanka_" in e.name}
    assert ran == {n[len("k_vanka_"):-1] for n in names}


@pytest.fixture(scope="module")
def large_tetra():
    P = problem("tetra", "one", 5)
    return P, Oracle(P)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("level", [2, 4])
def test_tetrahedra_on_both_sides_of_the_limits(large_tetra, precision, level):
    from to_merge_master_parmoon_gb300 import PmSolver
    P, O = large_tetra
    S = PmSolver(P.descs, precision=precision, restart=2)
    u, f = vectors(P, level)
    got, want = S.cell_vanka(level, u, f, 2), O.cell_vanka(level, u, f, 2)
    S.close()
    assert np.linalg.norm(got - want) < (1e-9 if precision == "fp64" else 5e-4) * np.linalg.norm(want)
