"""The modal sensor pass and the viscous terms on the active set, at every
degree, on ragged element counts (GPU vs oracle).

The states hold elements at rest, smooth and rough ones, so that the zero,
ramp and saturated branches of the sensor (and its tiny-energy branch) all
occur, in groups that cross the pass's warps (32 / n elements each) and end
in a partial one.

Bounds.  The viscosity is eps0 (1 + sin(x)) / 2 with x = pi (sigma - mid) /
width: log10 and sin are within an ulp of the oracle's, sigma is below 16 in
size, so x is off by at most 16 * 2^-52 * pi / width < 3e-15 (width >= 4) and
the viscosity by eps0 / 2 * (3e-15 + 2^-52 * 4) < 4e-15 eps0.  The right-hand
side is held to the bound of the other engine tests.
"""
import numpy as np
import pytest

from esdgsem_mpiocca_b200 import host
from esdgsem_mpiocca_b200.deviceclass import Solver
from oracle.oracle import OracleProblem
from tests.test_gpu_parity import assert_rhs_close

pytestmark = pytest.mark.gpu


def _rough(N, nx, ny, seed=0, **kw):
    args = dict(N=N, T=1e9, NumFlux=0, ArtificialViscosity=1, epsilon_0=0.01, sigma_min=-6.0, sigma_max=-2.0, DFL=0.1)
    args.update(kw)
    rng = np.random.default_rng(seed)
    m = host.mesh_mapped(N, 0.0, 1.0, 0.0, 1.0, nx, ny, amp=0.02, rotate_seed=3)
    n2 = (N + 1) ** 2
    q = np.zeros((m.K, 3, n2))
    amp = 10.0 ** rng.uniform(-7, -0.5, size=m.K)
    amp[::3] = 0.0
    q[:, 0] = 1.0 + amp[:, None] * rng.uniform(-1, 1, size=(m.K, n2))
    q[:, 1] = 0.1 * amp[:, None] * rng.uniform(-1, 1, size=(m.K, n2))
    q[m.K // 2, 0] = 1e-4                   # energy below the sensor's threshold
    b = np.zeros_like(m.x)
    return host.make_problem(host.Params(**args), m, b, q.reshape(-1))


def _check(pr, branches=True):
    s = Solver(pr)
    try:
        Qg, vg = s.rhs()
    finally:
        s.close()
    Qo, vo = OracleProblem(pr).rhs(pr.q0)
    eps0 = pr.params.epsilon_0
    if branches:
        assert (vo == 0).any() and ((vo > 0) & (vo < eps0)).any()
    np.testing.assert_array_equal(vg == 0, vo == 0)
    np.testing.assert_allclose(vg, vo, rtol=0, atol=4e-15 * eps0)
    assert_rhs_close(Qg, Qo, pr)


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("nx,ny", [(1, 1), (3, 5), (17, 15)])
def test_sensor_and_viscous_rhs(N, nx, ny):
    _check(_rough(N, nx, ny), branches=nx > 4 and N > 1)


@pytest.mark.parametrize("N", [2, 3, 4, 7])
def test_saturated_sensor(N):
    """sigma_max below the rough elements' sigma: viscosity eps0 there."""
    pr = _rough(N, 11, 9, sigma_min=-9.0, sigma_max=-5.0)
    _, vo = OracleProblem(pr).rhs(pr.q0)
    assert (vo == pr.params.epsilon_0).any()
    _check(pr)


@pytest.mark.parametrize("N", [3, 4, 6])
def test_every_element_viscous(N):
    pr = _rough(N, 13, 11, sigma_min=-60.0, sigma_max=-50.0)
    q = pr.q0.reshape(pr.K, 3, -1)
    q[:, 0] += 0.01 * np.random.default_rng(1).uniform(-1, 1, size=q[:, 0].shape)
    q[pr.K // 2, 0] += 1.0
    pr = host.make_problem(pr.params, pr.mesh, pr.b, pr.q0)
    _check(pr, branches=False)
