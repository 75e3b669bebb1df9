"""The chip-resident time loop where a block holds more nodes than threads
(GPU): the limiter's and the partial-dry treatment's flags then pass from one
pass over the elements to the next.  Against the step graph, bit for bit; and
loops of two solvers in two threads, against each alone.
"""
import threading

import numpy as np
import pytest

from esdgsem_mpiocca_b200.deviceclass import Solver
from tests.test_gpu_resident import _ragged, _run, _shore

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [
    lambda: _shore(1, 170, 171, False, 0),
    lambda: _shore(2, 112, 113, True, 1, rotate=3),
    lambda: _shore(3, 86, 87, False, 1),
    lambda: _shore(3, 96, 96, False, 1),
    lambda: _shore(4, 67, 69, True, 0, rotate=5),
    lambda: _shore(4, 70, 70, False, 1),
    lambda: _shore(7, 43, 45, False, 1),
], ids=["N1", "N2_ssp_dry", "N3_dry", "N3_dry_96", "N4_ssp", "N4_dry", "N7_dry"])
def test_limiter_over_several_passes(make):
    import torch
    prob = make()
    per_block = -(-prob.K // (2 * torch.cuda.get_device_properties(0).multi_processor_count))
    assert per_block * prob.ngl ** 2 > 384  # the larger block's threads
    g = _run(prob, True, 7)
    r = _run(prob, False, 7)
    assert r[4] <= 3 < g[4], "the resident loop did not run"
    assert r[0] == g[0]
    for a, b in zip(r[1:4], g[1:4]):
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, b)


def test_loops_in_two_threads():
    probs = [_ragged(4, 60, 61), _ragged(3, 40, 41, flux=2)]
    want, got, err = [], [None, None], []
    for pr in probs:
        s = Solver(pr)
        try:
            s.run(T=1e9, max_steps=200)
            want.append(s.q())
        finally:
            s.close()
    solvers = [Solver(pr) for pr in probs]

    def work(k):
        try:
            for _ in range(5):
                solvers[k].dc.copy_q_from_host(probs[k].q0)
                solvers[k].run(T=1e9, max_steps=200)
            got[k] = solvers[k].q()
        except Exception as e:
            err.append(e)

    try:
        ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    finally:
        for s in solvers:
            s.close()
    assert not err
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
