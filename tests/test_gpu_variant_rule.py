"""The element variant of a single mesh follows from its sizes and switches
(GPU), whatever the parity of its node count, and no kernel is launched to
find it.  Three kinds of mesh with a wide distance between the variants, measured:
with the partial-dry treatment the two-CTA kernel was 10 % faster than the
two-nodes-per-thread one, at N = 6 in the upper part of L2 and with viscosity
the latter 8 % and 3.5 % faster than the one-shot blocks.
"""
import dataclasses

import numpy as np
import pytest

from esdgsem_mpiocca_b200 import host, problems
from esdgsem_mpiocca_b200.deviceclass import Solver
from esdgsem_mpiocca_b200.ensemble import Ensemble

pytestmark = pytest.mark.gpu

TWO_CTAS, PAIR4 = 0, 6  # variants


def _lake(N, nel, **kw):
    pr = problems.curved_lake(N=N, nel=nel, seed=3, ripple=0.02)
    return host.make_problem(dataclasses.replace(pr.params, **kw), pr.mesh, pr.b, pr.q0, pr.meta)


@pytest.mark.parametrize("make,want", [
    (lambda: _lake(4, 127, PartialDryTreatment=1, PositivityPreserving=1), TWO_CTAS),
    (lambda: _lake(4, 128, PartialDryTreatment=1, PositivityPreserving=1), TWO_CTAS),
    (lambda: _lake(6, 115), PAIR4),
    (lambda: _lake(6, 116), PAIR4),
    (lambda: problems.dam_break(N=6, nel=91), PAIR4),
    (lambda: problems.dam_break(N=6, nel=92), PAIR4),
])
def test_variant_by_rule(make, want):
    s = Solver(make())
    try:
        assert s.dc.element_variants() is None
        l0 = s.dc.kernel_launches()
        s.run(T=1e9, max_steps=1)
        first = s.dc.kernel_launches() - l0
        ev = s.dc.element_variants()
        assert ev["chosen"] == want
        assert not np.any(ev["ms"])
        l0 = s.dc.kernel_launches()
        s.run(T=1e9, max_steps=1)
        assert s.dc.kernel_launches() - l0 == first
        assert np.isfinite(s.q()).all()
    finally:
        s.close()


def test_queries_only_read():
    """Asked from another thread all through a resident time loop, the variant
    queries give the choice or nothing, and the loop's result is that of a
    solver nobody asked."""
    import threading
    pr = problems.curved_lake(N=4, nel=20, seed=3, ripple=0.02)
    out, seen = {}, []
    for ask in (False, True):
        s = Solver(pr)
        stop = threading.Event()

        def watch():
            while not stop.is_set():
                seen.append((s.dc.element_variants(), s.dc.tuned_config()))

        t = threading.Thread(target=watch)
        try:
            if ask:
                t.start()
            first = s.run(T=1e9, max_steps=400)
            Q = s.rhs()
            out[ask] = (first, s.dc.advance(400, 1e9), Q, s.q())
            l0 = s.dc.kernel_launches()
            final = s.dc.element_variants()
            assert s.dc.kernel_launches() == l0 <= 8
        finally:
            stop.set()
            if ask:
                t.join()
            s.close()
    assert out[0][:2] == out[1][:2]
    np.testing.assert_array_equal(out[0][2], out[1][2])
    np.testing.assert_array_equal(out[0][3], out[1][3])
    assert seen and all(v is None or v == final for v, _ in seen)


def test_mostly_empty_arena_takes_no_one_shot_blocks():
    """Their grid covers the arena's capacity."""
    pr = problems.dam_break(N=1, nel=20)
    for slack, want in ((1.0, 7), (40.0, TWO_CTAS)):
        ens = Ensemble.for_problems([pr], slack=slack)
        try:
            i = ens.add(pr, T=1e9, max_steps=3)
            ens.advance(3)
            assert ens.element_variants()["chosen"] == want
            assert np.isfinite(ens.q(i)).all()
        finally:
            ens.close()
