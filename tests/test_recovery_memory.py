"""The scratch of a recovery: with it and without it the same bits, and a run takes none of the
memory that its own outputs or the caller's next buffers need."""
import gc

import numpy as np
import pytest

from femahoy_b200.recover import Recovery
from test_recovery import random_case

pytestmark = pytest.mark.gpu


def _new(c, nparts):
    return Recovery(c["xyz"], c["t10"], c["coef"], expansion=c["expansion"], part=c["part"],
                    nparts=nparts, singular=c["singular"])


def _same(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint8),
                          np.ascontiguousarray(b).view(np.uint8))


@pytest.mark.parametrize("dims,nparts", [((1, 1, 1), 1), ((7, 5, 3), 3), ((12, 9, 8), 70),
                                         ((19, 15, 7), 2), ((20, 10, 10), 3),
                                         ((34, 23, 22), 5)])
def test_points_that_evaluate_their_own_visits_give_the_same_bits(dims, nparts):
    """6 to 103,224 cells, with 11,970 and 12,000 at the line of 10 visits per thread."""
    c = random_case(dims, nparts=nparts)
    r = _new(c, nparts)
    for dtemp in (None, c["dtemp"]):
        for peaks in (True, False):
            want = r.with_scratch(4 << 30).run(c["u"], dtemp, peaks=peaks)
            got = r.with_scratch(640 * len(c["t10"]) - 1).run(c["u"], dtemp, peaks=peaks)
            for k in ("stress", "strain", "mises", "principal"):
                assert _same(got[k], want[k]), k
            if peaks:
                assert [vars(p) for p in got["peaks"]] == [vars(p) for p in want["peaks"]]


def test_scratch_leaves_room_for_the_outputs():
    """A device with room for the recovery and its outputs, or for the recovery and its scratch,
    but not for all three."""
    torch = pytest.importorskip("torch")
    c = random_case((46, 34, 32), nparts=3)
    r = _new(c, 3)
    want = r.run(c["u"], c["dtemp"])
    r.with_scratch(0).run(c["u"], c["dtemp"])  # both ways' kernels are loaded now
    need, scratch = r.bytes(), 640 * len(c["t10"])
    outputs = 8 * 20 * len(c["xyz"])
    del r
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    import femahoy_b200 as fg
    fg.trim()
    left = need + scratch - outputs + (30 << 20)
    assert left > need + (60 << 20)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        r = _new(c, 3)
        for _ in range(2):
            assert _same(r.run(c["u"], c["dtemp"])["stress"], want["stress"])
    finally:
        del hold
        torch.cuda.empty_cache()


def test_threads_side_by_side_give_the_same_bits():
    """Each run takes its scratch from the pool that all of them share."""
    from concurrent.futures import ThreadPoolExecutor
    cases = [random_case(d, nparts=2) for d in ((9, 7, 5), (20, 10, 10), (14, 9, 8), (24, 11, 9))]
    made = [_new(c, 2) for c in cases]
    alone = [r.run(c["u"], c["dtemp"]) for r, c in zip(made, cases)]

    def again(k):
        return [made[k].run(cases[k]["u"], cases[k]["dtemp"]) for _ in range(6)]

    with ThreadPoolExecutor(max_workers=len(made)) as pool:
        for want, runs in zip(alone, pool.map(again, range(len(made)))):
            for got in runs:
                for k in ("stress", "strain", "mises", "principal"):
                    assert _same(got[k], want[k]), k
