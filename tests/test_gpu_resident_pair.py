"""Several solvers whose time loops run in the same instance of the
chip-resident kernel (GPU): each keeps its loop, whatever the others' sizes
and the order in which they were built.  A run in it is three launches at
most (bottom traces, wave speed, the loop), in the step graph more than that
for every step.
"""
import numpy as np
import pytest

from esdgsem_mpiocca_b200.deviceclass import Solver
from tests.test_gpu_resident import _ragged, _shore

pytestmark = pytest.mark.gpu

STEPS = 6


def _launches(s):
    l0 = s.dc.kernel_launches()
    s.run(T=1e9, max_steps=STEPS)
    return s.dc.kernel_launches() - l0


@pytest.mark.parametrize("makes", [
    # one degree, one block size: the largest first, so that a smaller one is
    # built after it
    [lambda: _ragged(4, 88, 94), lambda: _ragged(4, 64, 64), lambda: _ragged(4, 60, 61)],
    [lambda: _ragged(3, 16, 16), lambda: _ragged(3, 5, 3)],
    [lambda: _shore(3, 96, 96, False, 1), lambda: _shore(3, 70, 70, False, 1), lambda: _shore(3, 70, 70, True, 0)],
    [lambda: _shore(1, 160, 160, False, 0), lambda: _shore(1, 40, 37, False, 0)],
], ids=["plain_N4", "plain_N3", "shore_N3", "shore_N1"])
def test_each_solver_keeps_its_loop(makes):
    probs = [m() for m in makes]
    alone = []
    for pr in probs:
        s = Solver(pr)
        try:
            assert _launches(s) <= 3
            alone.append(s.q())
        finally:
            s.close()
    solvers = [Solver(pr) for pr in probs]
    try:
        for order in (range(len(solvers)), reversed(range(len(solvers)))):
            for k in order:
                solvers[k].dc.copy_q_from_host(probs[k].q0)
                assert _launches(solvers[k]) <= 3, k
                np.testing.assert_array_equal(solvers[k].q(), alone[k])
    finally:
        for s in solvers:
            s.close()
