"""Vanka sweeps from packed rows (the default on one-block hexahedral levels)
against the CSR kernels (residual_variant=1), on every level of several
meshes: cubes, boxes with odd cell counts, a level of one cell per direction,
a periodic stretched channel, and a random numbering of the velocity nodes (no
two cells share a pattern).

FP32: both run the same operations in the same order, so the sweeps are equal
bit for bit.  FP64: the sums run in another order; two sweeps of condition
O(10) amplify 2e-16 to well below 1e-12."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MESHES = {
    "cube": dict(n_levels=4),
    "box": dict(n_levels=3, nx0=3, ny0=2, nz0=1, box=(0, 1.5, 0, 1, 0, 0.5)),
    "one_cell": dict(n_levels=2, nx0=1, ny0=1, nz0=1),
    "channel": dict(n_levels=3, nx0=4, ny0=3, nz0=2, example="channel", periodic="xz",
                    stretch_y=2.0, box=(0, 6.28, -1, 1, 0, 3.14)),
}


def shuffled(P, seed):
    """The levels of P with their active velocity nodes renumbered at random;
    returns (descriptors, arrays kept alive, new number of each node)."""
    from to_merge_master_parmoon_gb300._lib import PmLevelDesc
    rng = np.random.default_rng(seed)
    descs, keep, perms = (PmLevelDesc * P.n_levels)(), [], []
    for lev in range(P.n_levels):
        a = P.arrays(lev)
        nu, na = a["n_udof"], a["n_active"]
        new = np.arange(nu)
        new[:na] = rng.permutation(na)
        old = np.argsort(new)
        C.pointer(descs[lev])[0] = P.desc(lev)
        d = descs[lev]

        def put(name, arr, index=None):
            keep.append(arr)
            typ = C.c_int if arr.dtype == np.int32 else C.c_double
            ptr = arr.ctypes.data_as(C.POINTER(typ))
            if index is None:
                setattr(d, name, ptr)
            else:
                getattr(d, name)[index] = ptr

        def rows(prefix, col_new, row_old):
            """Rows in the order row_old, columns through col_new, sorted."""
            rp, col = a[prefix + "_rowptr"], a[prefix + "_col"]
            n = np.diff(rp)[row_old]
            nrp = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
            src = np.repeat(rp[row_old], n) + np.arange(nrp[-1]) - np.repeat(nrp[:-1], n)
            c = col[src] if col_new is None else col_new[col[src]]
            order = np.lexsort((c, np.repeat(np.arange(len(n)), n)))
            put(prefix + "_rowptr", nrp)
            put(prefix + "_col", c[order].astype(np.int32))
            for k, v in enumerate(a[prefix]):
                put(prefix, np.ascontiguousarray(v[src][order]), k)

        rows("a", new, old)
        rows("b", new, np.arange(a["n_pdof"]))
        rows("bt", None, old)
        put("cell_udofs", np.ascontiguousarray(new[a["cell_udofs"]].astype(np.int32)))
        perms.append(new)
    return descs, keep, perms


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("mesh", list(MESHES))
def test_equal_to_the_csr_kernels(mesh, precision):
    from to_merge_master_parmoon_gb300 import OseenProblem, PmSolver
    P = OseenProblem(nu=1e-2, seed=3, **MESHES[mesh])
    A = PmSolver(P.descs, precision=precision)
    B = PmSolver(P.descs, precision=precision, residual_variant=1)
    rng = np.random.default_rng(0)
    for level in range(1, P.n_levels):
        u, f = 0.1 * rng.standard_normal(P.ndof(level)), rng.standard_normal(P.ndof(level))
        for sweeps in (1, 2, 3):
            a, b = A.cell_vanka(level, u, f, sweeps), B.cell_vanka(level, u, f, sweeps)
            if precision == "mixed":
                assert np.array_equal(a, b)
            else:
                assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)
    A.close()
    B.close()


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("alpha", [1.0, 0.7])
def test_any_numbering(precision, alpha):
    """Random numbering, with and without level relaxation: packed and CSR
    sweeps agree as above, and renumbered back they agree with the original
    numbering to the precision of the sweep."""
    from to_merge_master_parmoon_gb300 import OseenProblem, PmSolver
    P = OseenProblem(n_levels=3, nu=1e-2, seed=4)
    descs, keep, perms = shuffled(P, 7)
    A = PmSolver(descs, precision=precision, alpha=alpha)
    B = PmSolver(descs, precision=precision, alpha=alpha, residual_variant=1)
    S = PmSolver(P.descs, precision=precision, alpha=alpha)
    rng = np.random.default_rng(1)
    for level in (1, 2):
        nu, new = P.desc(level).n_udof, perms[level]
        u, f = 0.1 * rng.standard_normal(P.ndof(level)), rng.standard_normal(P.ndof(level))

        def move(v):
            w = v.copy()
            for k in range(3):
                w[k * nu + new] = v[k * nu:(k + 1) * nu]
            return w

        a, b = A.cell_vanka(level, move(u), move(f), 2), B.cell_vanka(level, move(u), move(f), 2)
        s = move(S.cell_vanka(level, u, f, 2))
        if precision == "mixed":
            assert np.array_equal(a, b)
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)
        assert np.linalg.norm(a - s) <= (1e-5 if precision == "mixed" else 1e-12) * np.linalg.norm(s)
    for h in (A, B, S):
        h.close()


def test_packed_rows_yield_to_other_allocations():
    """Under a memory cap the packed copy is not made when it does not fit and
    given back when a later allocation needs the room; results stay."""
    from to_merge_master_parmoon_gb300 import OseenProblem, PmSolver
    P = OseenProblem(n_levels=3, nu=1e-2, seed=3)
    b = P.rhs()
    S = PmSolver(P.descs, precision="mixed")
    need, want = S.device_bytes, S.vcycle(b)
    S.close()
    conv = [P.convection_nodal(k) for k in range(3)]
    for extra in (0, 1 << 22, 1 << 24):
        S = PmSolver(P.descs, precision="mixed", max_device_bytes=need + extra)
        assert np.array_equal(S.vcycle(b), want)
        if extra:  # the assembly's own buffers evict the copy where they have to
            for k in range(3):
                S.assemble_level(k, P.cell_sizes(k), conv[k], P.nu)
            S.refactor()
            got = S.vcycle(b)
            assert np.linalg.norm(got - want) <= 5e-4 * np.linalg.norm(want)
        S.close()


def test_new_values_reach_the_sweeps():
    """Matrices assembled again with another viscosity: sweeps with and
    without a refactorisation in between use the new rows (FP32, equal to the
    CSR kernels)."""
    from to_merge_master_parmoon_gb300 import OseenProblem, PmSolver
    P = OseenProblem(n_levels=3, nu=1e-2, seed=3)
    A = PmSolver(P.descs, precision="mixed")
    B = PmSolver(P.descs, precision="mixed", residual_variant=1)
    rng = np.random.default_rng(2)
    u, f = 0.1 * rng.standard_normal(P.ndof(2)), rng.standard_normal(P.ndof(2))
    for nu in (3e-2, 5e-3):
        for S in (A, B):
            for k in range(3):
                S.assemble_level(k, P.cell_sizes(k), P.convection_nodal(k), nu)
        assert np.array_equal(A.cell_vanka(2, u, f, 2), B.cell_vanka(2, u, f, 2))
        for S in (A, B):
            S.refactor()
        assert np.array_equal(A.cell_vanka(2, u, f, 2), B.cell_vanka(2, u, f, 2))
        assert np.array_equal(A.vcycle(f), B.vcycle(f))
    A.close()
    B.close()
