"""The stress recovery at the sizes where its rules change (2 visits per thread, then a cell's 10),
bit for bit against the oracle, with and without temperatures and peaks."""
import numpy as np
import pytest

import oracle
from femahoy_b200.recover import Recovery
from test_recovery import oracle_of, random_case

pytestmark = pytest.mark.gpu


def _same(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint8),
                          np.ascontiguousarray(b).view(np.uint8))


@pytest.mark.parametrize("dims,nparts", [((1, 1, 1), 1), ((7, 5, 3), 3), ((34, 22, 22), 70),
                                         ((34, 23, 22), 5)])
def test_bits(dims, nparts):
    """6, 630, 98,736 cells (2 visits per thread; 70 parts keep their maxima in global memory)
    and 103,224 (10)."""
    c = random_case(dims, nparts=nparts)
    want = oracle_of(c)
    r = Recovery(c["xyz"], c["t10"], c["coef"], expansion=c["expansion"], part=c["part"],
                 nparts=nparts, singular=c["singular"])
    got = r.run(c["u"], c["dtemp"])
    for k in ("stress", "strain", "mises"):
        assert _same(got[k], want[k]), k
    bare = r.run(c["u"], c["dtemp"], peaks=False, principal=False)
    assert bare["peaks"] is None and _same(bare["stress"], want["stress"])
    for p, q in zip(got["peaks"], want["peaks"]):
        assert (p.mises, p.element, p.local, p.regular_element) == (
            q.mises, q.element, q.local, q.regular_element)
    cold = oracle.recover(c["xyz"], c["t10"], c["coef"], c["u"], expansion=c["expansion"],
                          part=c["part"], nparts=nparts, singular=c["singular"])
    assert _same(r.run(c["u"], peaks=False)["stress"], cold["stress"])
