"""Choosing the element variant again leaves the solution alone (GPU).

A viscous loop that ends by T, by a pause or by the step cap leaves the flags
of its last sensor pass set.  Giving the variant choice back to the engine
(-1) after that must not change the state: the further steps are those of a
solver whose variant was never touched, bit for bit (all variants compute the
same bits), at the sizes where the flagged elements would fill the active
set's list many times over.
"""
import numpy as np
import pytest

from esdgsem_mpiocca_b200 import problems
from esdgsem_mpiocca_b200.deviceclass import Solver
from esdgsem_mpiocca_b200.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def _viscous(N, nel):
    pr = problems.dam_break(N=N, nel=nel, seed=1)
    assert pr.params.ArtificialViscosity
    return pr


@pytest.mark.parametrize("N,nel", [(3, 20), (4, 24), (6, 9)])
@pytest.mark.parametrize("by", ["T", "pause", "cap"])
@pytest.mark.parametrize("then", ["profile", "advance"])
def test_viscous_run_after_choosing_again(N, nel, by, then):
    import torch
    out = {}
    for again in (False, True):
        s = Solver(_viscous(N, nel))
        stream = torch.cuda.Stream()
        try:
            t1, n1 = s.run(T=1e9, max_steps=9)
            if by == "T":
                t, n = s.run(T=0.6 * t1)
            elif by == "pause":
                assert s.dc._L.esdg_set_pause(s.dc.h, 0.5 * t1) == 0
                t, n = s.run(T=10 * t1)
                assert s.dc._L.esdg_set_pause(s.dc.h, float("inf")) == 0
            else:
                t, n = t1, n1
            assert np.count_nonzero(s.dc.copy_visc_to_host(s.prob.K)) * 30 > s.prob.K
            before = s.q()
            if again:
                s.dc.set_element_variant(-1)
            if then == "profile":
                s.dc.profile_steps(2)
            else:
                s.dc.set_stream(stream.cuda_stream)
                s.dc.advance(2, 1e9)
            out[again] = (t, n, before, s.q())
        finally:
            s.close()
    assert out[0][:2] == out[1][:2]
    for a, b in zip(out[1][2:], out[0][2:]):
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, b)
    # a paused loop's further steps wait for resume: q stays as it was
    assert np.array_equal(out[0][2], out[0][3]) == (by == "pause")


def test_viscous_ensemble_after_choosing_again():
    probs = [_viscous(3, 12), _viscous(3, 9)]
    out = {}
    for again in (False, True):
        ens = Ensemble.for_problems(probs)
        try:
            ids = [ens.add(p, T=1e9, max_steps=m) for p, m in zip(probs, (4, 12))]
            ens.advance(6)  # the first ends, the second is in the middle
            if again:
                ens.set_element_variant(-1)
            ens.advance(6)
            out[again] = [ens.q(i) for i in ids]
        finally:
            ens.close()
    for a, b in zip(out[1], out[0]):
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, b)
