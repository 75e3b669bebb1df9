"""Element kernels on meshes with an odd number of nodes (GPU).

An odd element count times an odd n^2 ends in a tile whose bulk copies are
not whole 16-byte words; they are rounded up into the buffers' padding.
Every variant must give the same bits as the others, the right-hand side of
the oracle within the engine tests' bound, and time steps equal to the
chip-resident loop's (which copies nothing in bulk).
"""
import numpy as np
import pytest

from esdgsem_mpiocca_b200 import host, problems
from esdgsem_mpiocca_b200.deviceclass import Solver
from oracle.oracle import OracleProblem
from tests.test_gpu_parity import assert_rhs_close

pytestmark = pytest.mark.gpu


def _mesh(N, nx, ny):
    m = host.mesh_mapped(N, 0.0, 1.0, 0.0, 1.0, nx, ny, amp=0.03, rotate_seed=5)
    b = problems.gaussian_bumps(m.x, m.y, 2)
    q = np.zeros((m.K, 3, (N + 1) ** 2))
    q[:, 0] = (1.0 - b + 0.05 * np.sin(9 * m.x) * np.cos(7 * m.y)).reshape(m.K, -1)
    q[:, 2] = (0.1 * np.cos(5 * m.x)).reshape(m.K, -1)
    return host.make_problem(host.Params(N=N, T=1e9, NumFlux=0), m, b, q.reshape(-1))


@pytest.mark.parametrize("N,nx,ny", [(2, 1, 1), (2, 29, 1), (2, 31, 29), (4, 1, 9), (4, 11, 1), (4, 21, 13), (6, 1, 3),
                                     (6, 5, 7), (6, 13, 11)])
def test_every_variant_on_odd_node_counts(N, nx, ny):
    pr = _mesh(N, nx, ny)
    assert pr.K * (N + 1) ** 2 % 2 == 1
    s = Solver(pr)
    try:
        s.run(T=1e9, max_steps=5)
        resident = s.q()
        usable = [v for v, c in enumerate(s.dc.element_variants()["ctas_per_sm"]) if c > 0]
    finally:
        s.close()
    Qo = OracleProblem(pr).rhs(pr.q0)
    Qo = Qo[0] if isinstance(Qo, tuple) else Qo
    for v in usable:
        s = Solver(pr)
        try:
            s.dc.set_element_variant(v)
            assert_rhs_close(s.rhs(), Qo, pr)
            s.run(T=1e9, max_steps=5)
            np.testing.assert_array_equal(s.q(), resident, err_msg=f"variant {v}")
        finally:
            s.close()
