"""The bounded waits of the chip-resident time loop (GPU).

Its thread blocks wait for their neighbours' traces with a clock-cycle limit.
A test hook sets the limit to one cycle -- nothing faults: the first waits run
out (a trace takes a thousand cycles or more), every block returns, and the
run reports ESDG_E_CUDA with a message of its own and leaves q alone.  The
same solver then runs, hook off, to the step graph's result, bit for bit.
"""
import numpy as np
import pytest

from esdgsem_mpiocca_b200 import problems
from esdgsem_mpiocca_b200.deviceclass import E_UNSUPPORTED, EsdgError, Solver
from tests.test_gpu_resident import _ragged, _shore

pytestmark = pytest.mark.gpu

E_CUDA = -3
LIMIT = 1


@pytest.mark.parametrize("make", [
    lambda: _ragged(3, 16, 16),              # small block, words sent with the update
    lambda: _ragged(4, 64, 64),              # large block
    lambda: _shore(3, 41, 40, False, 1),     # limiter and partial-dry treatment
    lambda: problems.periodic_bump(N=2, nel=3, NumFlux=0),
])
def test_wait_runs_out_and_solver_stays_usable(make):
    pr = make()
    ref = Solver(pr)
    try:
        ref.dc.debug_bulk_wait_test(4_000_000_000, -1)  # the step graph
        want = ref.run(T=1e9, max_steps=5) + (ref.q(),)
    finally:
        ref.close()
    s = Solver(pr)
    try:
        s.run(T=1e9, max_steps=2)
        before = s.q()
        s.dc.debug_resident_wait_test(LIMIT)
        l0 = s.dc.kernel_launches()
        with pytest.raises(EsdgError) as ei:
            s.run(T=1e9, max_steps=5)
        assert s.dc.kernel_launches() - l0 <= 3
        assert ei.value.code == E_CUDA
        assert "bounded wait" in str(ei.value) and "bulk copy" not in str(ei.value)
        np.testing.assert_array_equal(s.q(), before)
        with pytest.raises(EsdgError) as ei:
            s.dc.advance(2, 1e9)
        assert ei.value.code == E_CUDA
        s.dc.debug_resident_wait_test(0)
        s.dc.copy_q_from_host(pr.q0)
        got = s.run(T=1e9, max_steps=5)
        assert got == want[:2]
        np.testing.assert_array_equal(s.q(), want[2])
    finally:
        s.close()


def test_hook_is_refused_where_it_reaches_nothing():
    s = Solver(problems.dam_break(N=3, nel=8))  # viscosity: the step graph
    try:
        with pytest.raises(EsdgError) as ei:
            s.dc.debug_resident_wait_test(LIMIT)
        assert ei.value.code == E_UNSUPPORTED
    finally:
        s.close()
    s = Solver(_ragged(3, 4, 4))
    try:
        with pytest.raises(EsdgError):
            s.dc.debug_resident_wait_test(-1)
    finally:
        s.close()
