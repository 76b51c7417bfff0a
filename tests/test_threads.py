"""Handles of several host threads: each thread factors a handle of its own
(one handle belongs to one thread at a time, several handles run at once).
The coarse systems have 2,443, 1,137 and 407 unknowns, so their LU panels ask
for different amounts of shared memory.  No call fails, and the coarse solves
agree bit for bit with those of the same handle before the threads started."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_factorisations_of_several_threads():
    from to_merge_master_parmoon_gb300 import OseenProblem, PmSolver
    problems = [OseenProblem(n_levels=1, nu=1e-2, seed=1, nx0=n, ny0=n, nz0=n) for n in (4, 3, 2)]
    handles = [PmSolver(P.descs) for P in problems]
    rhs = [np.random.default_rng(k).standard_normal(P.ndof(0)) for k, P in enumerate(problems)]
    want = [S.solve_exact(b) for S, b in zip(handles, rhs)]
    errors = []

    def work(S, b, x, times):
        try:
            for _ in range(times):
                S.refactor()
            assert np.array_equal(S.solve_exact(b), x)
        except Exception as e:  # noqa: BLE001 - handed to the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(S, b, x, n))
               for S, b, x, n in zip(handles, rhs, want, (20, 60, 150))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for S in handles:
        S.close()
    assert not errors
