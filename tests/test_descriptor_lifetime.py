"""One-block descriptors share the arrays of their problem: they have to keep
it alive (a cache that dropped the problem first left dangling row pointers)."""
import gc
import weakref

import numpy as np


def test_one_block_descriptors_keep_their_problem():
    from to_merge_master_parmoon_gb300 import OseenProblem
    P = OseenProblem(n_levels=2, nu=1e-2, seed=0)
    want = [P.desc(level).a_nnz for level in range(2)]
    alive, D = weakref.ref(P), P.descs_one_block()
    del P
    gc.collect()
    assert alive() is not None
    got = [int(np.ctypeslib.as_array(D[k].a_rowptr, shape=(D[k].n_udof + 1,))[-1]) for k in range(2)]
    assert got == want
    del D
    gc.collect()
    assert alive() is None
