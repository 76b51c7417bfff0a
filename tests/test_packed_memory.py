"""The packed copy of the matrix rows is optional: it is reported apart from the
memory a handle needs, given back level by level to allocations that need the
room, made again when there is room, and not made where it would leave less
than half of the device free.  Results stay (FP32 bit for bit)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# packed bytes of a cell in FP32: rows and patch list (the other arrays are small)
CELL = 4 * (3904 + 400)


def test_levels_are_given_back_one_by_one():
    from to_merge_master_parmoon_gb300 import OseenProblem, PmSolver
    P = OseenProblem(n_levels=4, nu=1e-2, seed=3)  # 64, 512 and 4,096 cells in smoothed levels
    b = P.rhs()
    S = PmSolver(P.descs, precision="mixed")
    need, packed, want = S.device_bytes, S.packed_bytes, S.vcycle(b)
    assert packed > CELL * (64 + 512 + 4096)
    S.close()
    # room for all of it, but not for the buffers of an assembly as well
    S = PmSolver(P.descs, precision="mixed", max_device_bytes=need + packed)
    assert S.packed_bytes == packed
    for k in range(2):  # small buffers of the two coarsest levels
        S.assemble_level(k, P.cell_sizes(k), P.convection_nodal(k), P.nu)
    kept = S.packed_bytes
    assert CELL * 4096 < kept < packed  # the finest level keeps its copy
    S.refactor()
    got = S.vcycle(b)
    assert np.linalg.norm(got - want) <= 5e-4 * np.linalg.norm(want)
    S.close()


def test_made_again_and_not_beyond_half_of_the_device():
    import torch
    from to_merge_master_parmoon_gb300 import OseenProblem, PmSolver
    P = OseenProblem(n_levels=3, nu=1e-2, seed=3)
    b = P.rhs()
    free, total = torch.cuda.mem_get_info()
    hold = torch.empty(max(0, free - int(0.45 * total)), dtype=torch.uint8, device="cuda")
    S = PmSolver(P.descs, precision="mixed")
    assert S.packed_bytes == 0
    without = S.vcycle(b)
    del hold
    torch.cuda.empty_cache()
    assert S.packed_bytes == 0
    S.refactor()
    assert S.packed_bytes > CELL * (64 + 512)
    assert np.array_equal(S.vcycle(b), without)
    S.close()
