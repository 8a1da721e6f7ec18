"""Solves of several host threads at once (pm_coop.cu): the cooperative kernels of
different handles share the SMs instead of waiting for one another."""
import threading
import time

import numpy as np
import pytest

import poromec_gb300 as pg
from poromec_gb300 import meshgen

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

THREADS, SOLVES = 4, 8


# a warp per node, and two nodes per warp
@pytest.mark.parametrize("n", [5, 11])
def test_four_threads_keep_the_phase_kernels_rate(n, monkeypatch):
    """Four threads with a handle each, against the same through the phase kernels,
    whose launches interleave. Two cooperative solves at a time take 0.95 to 1.05
    of that, one after the other 1.6 to 1.8: at most 1.3, best of three runs each."""
    pb = meshgen.cube_problem(n=n)
    ms, rhs, sol = [], [], []
    for k in range(THREADS):
        m = pg.from_problem(pb)
        m.pform(2, True, False, np.zeros((m.nnode, 4)), None)
        ms.append(m)
        rhs.append(torch.from_numpy(np.random.default_rng(k).standard_normal(m.neq)).cuda())
        sol.append(torch.zeros_like(rhs[-1]))
    torch.cuda.synchronize()

    def work(k):
        for _ in range(SOLVES):
            ms[k].solve_dev(rhs[k].data_ptr(), sol[k].data_ptr(), solver=1, precond=2, tol=1e-10,
                            maxit=20000)

    def best():
        times = []
        for _ in range(4):  # the first warms up
            ts = [threading.Thread(target=work, args=(k,)) for k in range(THREADS)]
            t0 = time.perf_counter()
            for t in ts:
                t.start()
            for t in ts:
                t.join()
            times.append(time.perf_counter() - t0)
        return min(times[1:])

    work(0)
    alone = sol[0].clone()
    coop = best()
    assert torch.equal(sol[0], alone)  # and the solution does not depend on the others
    monkeypatch.setenv("PM_POLLED_GRAPHS", "1")
    assert coop <= 1.3 * best()
