"""The chip-resident time loop against the step graph (GPU).

A small plain mesh runs its steps inside one kernel (esdg_resident.cu); the
step graph runs the same steps kernel by kernel.  Both do the same
operations in the same order on every node, so the states, the times and
the RK register's effect on further steps must be equal exactly.  The step
graph is selected by naming the default wait limit explicitly (the bulk-wait
hook concerns its kernels only).
"""
import dataclasses

import numpy as np
import pytest

from esdgsem_mpiocca_b200 import host, problems
from esdgsem_mpiocca_b200.deviceclass import Solver

pytestmark = pytest.mark.gpu


def _with(prob, ssp=False, **kw):
    if ssp:
        kw.update(rkOrder=3, rkSSP=1)
    p = dataclasses.replace(prob.params, **kw)
    return host.make_problem(p, prob.mesh, prob.b, prob.q0, prob.meta)


def _shore(N, nx, ny, ssp, pd, rotate=0):
    """A lake around an island above the surface: h = 0 nodes, limiter on."""
    p = host.Params(N=N, CFL=0.3, T=1e9, NumFlux=0, PositivityPreserving=1, PosPresTOL=1e-3, PartialDryTreatment=pd,
                    rkOrder=3 if ssp else 4, rkSSP=int(ssp))
    m = host.mesh_mapped(N, 0.0, 1.0, 0.0, 1.0, nx, ny, amp=0.02, rotate_seed=rotate)
    b = 1.4 * np.exp(-((m.x - 0.47) ** 2 + (m.y - 0.52) ** 2) / 0.18 ** 2)
    wet = np.maximum(0.0, 1.0 - b)
    h = np.where(wet > 0, wet + 0.05 * np.exp(-((m.x - 0.7) ** 2 + (m.y - 0.3) ** 2) / 0.1 ** 2), 0.0)
    q = np.zeros((m.K, 3, (N + 1) ** 2))
    q[:, 0] = h.reshape(m.K, -1)
    return host.make_problem(p, m, b, q.reshape(-1))


def _ragged(N, nx, ny, flux=0, rotate=3):
    """nx x ny curved elements (odd counts allowed), ripple over a bump."""
    p = host.Params(N=N, T=1e9, NumFlux=flux)
    m = host.mesh_mapped(N, 0.0, 1.0, 0.0, 1.0, nx, ny, amp=0.03, rotate_seed=rotate)
    b = problems.gaussian_bumps(m.x, m.y, 5)
    q = np.zeros((m.K, 3, (N + 1) ** 2))
    q[:, 0] = (1.0 - b + 0.05 * np.sin(9 * m.x) * np.cos(7 * m.y)).reshape(m.K, -1)
    q[:, 1] = (0.1 * np.sin(5 * m.y)).reshape(m.K, -1)
    return host.make_problem(p, m, b, q.reshape(-1))


CASES = {
    "N1_one_column": lambda: _ragged(1, 1, 7),
    "N1_many": lambda: _ragged(1, 151, 97, flux=3),
    "N2_ssp": lambda: _with(_ragged(2, 13, 11, flux=2), ssp=True),
    "N3_periodic_strip": lambda: problems.periodic_bump(N=3, nel=2, NumFlux=2),
    "N3_periodic": lambda: problems.periodic_bump(N=3, nel=16, NumFlux=0),
    "N3_one_pass": lambda: _ragged(3, 64, 74, flux=2),       # 32 elements a CTA: one full pass of 512 threads
    "N3_two_passes": lambda: _ragged(3, 64, 77, flux=3),     # 34: the second pass holds two
    "N4_odd": lambda: _ragged(4, 33, 31),
    "N4_largest": lambda: _ragged(4, 88, 94),                # close to what the shared memory holds
    "N5_rot": lambda: _ragged(5, 19, 23, flux=3, rotate=11),
    "N6_odd_nodes": lambda: _ragged(6, 21, 21),
    "N7": lambda: _ragged(7, 30, 25, flux=3),
    "shore_N1": lambda: _shore(1, 40, 37, False, 0),
    "shore_ssp_N2": lambda: _shore(2, 33, 29, True, 0, rotate=7),
    "shore_dry_N3": lambda: _shore(3, 41, 40, False, 1),
    "shore_dry_ssp_N4": lambda: _shore(4, 20, 23, True, 1, rotate=2),
    "shore_N7": lambda: _shore(7, 12, 9, False, 0),
}


def _run(prob, graph, steps):
    s = Solver(prob)
    try:
        if graph:
            s.dc.debug_bulk_wait_test(4_000_000_000, -1)
        l0 = s.dc.kernel_launches()
        t1, n1 = s.run(T=1e9, max_steps=steps)
        launches = s.dc.kernel_launches() - l0
        qa = s.q()
        t2, n2 = s.dc.advance(3, 1e9)
        qb = s.q()
        t3, n3 = s.dc.advance(100, t2 + 0.4 * (t2 - t1) / 3)  # ends at T, within a step
        return (t1, n1, t2, n2, t3, n3), qa, qb, s.q(), launches
    finally:
        s.close()


@pytest.mark.parametrize("name", list(CASES))
def test_resident_loop_equals_step_graph(name):
    prob = CASES[name]()
    steps = 7
    g = _run(prob, True, steps)
    r = _run(prob, False, steps)
    assert r[4] <= 3 < g[4], "the resident loop did not run"  # bottom traces, wave speed, the loop
    assert r[0] == g[0]
    for a, b in zip(r[1:4], g[1:4]):
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, b)


def test_pause_and_resume_equal_step_graph():
    out = {}
    for graph in (False, True):
        s = Solver(problems.periodic_bump(N=3, nel=10, NumFlux=0))
        try:
            if graph:
                s.dc.debug_bulk_wait_test(4_000_000_000, -1)
            L = s.dc._L
            assert L.esdg_set_pause(s.dc.h, 0.01) == 0
            first = s.run(T=0.03, max_steps=0)
            assert L.esdg_set_pause(s.dc.h, float("inf")) == 0
            import ctypes
            t, n = ctypes.c_double(), ctypes.c_int()
            assert L.esdg_resume(s.dc.h, ctypes.byref(t), ctypes.byref(n)) == 0
            out[graph] = (first, t.value, n.value, s.q())
        finally:
            s.close()
    assert out[0][:3] == out[1][:3]
    np.testing.assert_array_equal(out[0][3], out[1][3])


def test_loop_that_ends_in_a_later_launch():
    """More steps than one launch holds (1024), ended by the step cap."""
    res = {}
    for graph in (False, True):
        s = Solver(problems.periodic_bump(N=1, nel=4, NumFlux=0))
        try:
            if graph:
                s.dc.debug_bulk_wait_test(4_000_000_000, -1)
            res[graph] = s.run(T=1e9, max_steps=1500) + (s.q(),)
        finally:
            s.close()
    assert res[0][:2] == res[1][:2] and res[0][1] == 1500
    np.testing.assert_array_equal(res[0][2], res[1][2])
