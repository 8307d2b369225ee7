"""The evaluation's schedule with many queries to one group.

A group's queries are cut into units of up to 512; the schedule places all units
of all groups before the evaluation starts.  Each query's value is the same in
whatever company it is asked (the partial sums of a unit that is cut between
blocks meet in another order: a few of 52 bits, 1e-12 absolute on the logarithm),
and many queries to one group take no longer than as many spread over groups of
as many points: the terms to sum are the same, so 1.3 leaves the clock's noise.
"""

import numpy as np
import pytest
import torch

from ssms_b200 import kde as gk

pytestmark = pytest.mark.gpu


def _fit(sizes, seed=1):
    rng = np.random.default_rng(seed)
    n = int(np.sum(sizes))
    rts = torch.from_numpy(np.exp(rng.normal(0.0, 0.5, n)).astype(np.float32))
    return gk.KdeBatch(rts, torch.ones(n, dtype=torch.int32), np.concatenate([[0], np.cumsum(sizes)]), [1]), rng


@pytest.mark.parametrize("n_q", [
    [0, 5, 513 * 1024 + 7, 0, 300, 0],      # one group with more units than the scheduling block has threads
    [1, 0, 0, 512, 512 * 1024, 1],          # whole units only
    [3] * 1500 + [40_000] + [0] * 700 + [1025, 0],  # several scans of 1 024 groups
])
def test_values_do_not_depend_on_the_other_queries(cuda, n_q):
    sizes = [(37 * i) % 90 + 1 if i % 5 else 0 for i in range(len(n_q))]
    big = int(np.argmax(n_q))
    sizes[big] = 700
    kb, rng = _fit(sizes)
    qoff = np.concatenate([[0], np.cumsum(n_q)]).astype(np.int64)
    q = torch.from_numpy(np.exp(rng.normal(0.0, 0.6, int(qoff[-1])))).cuda()
    got = kb.evaluate(qoff, q, max_t=20.0).cpu().numpy()
    step = 20_000
    pieces = [(g, a, min(a + step, int(qoff[g + 1]))) for g in (big, len(n_q) - 2, 0)
              for a in range(int(qoff[g]), int(qoff[g + 1]), step)]
    for g, a, b in pieces:
        part = np.where(np.arange(len(n_q) + 1) > g, b - a, 0).astype(np.int64)
        want = kb.evaluate(part, q[a:b], max_t=20.0).cpu().numpy()
        np.testing.assert_allclose(got[a:b], want, rtol=0, atol=1e-12)


def _time(f):
    f()
    ms = []
    for _ in range(7):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        f()
        e1.record()
        torch.cuda.synchronize()
        ms.append(e0.elapsed_time(e1))
    return min(ms)


def test_many_queries_to_one_group_cost_no_more_than_to_many(cuda):
    one, rng = _fit([1000])
    many, _ = _fit([1000] * 1000)
    q = torch.from_numpy(np.exp(rng.normal(0.0, 0.6, 1_000_000))).cuda()
    o1, om = torch.tensor([0, 1_000_000]), torch.arange(0, 1_000_001, 1000)
    o1, om = o1.cuda(), om.cuda()
    t1 = _time(lambda: one.evaluate(o1, q, max_t=20.0))
    tm = _time(lambda: many.evaluate(om, q, max_t=20.0))
    assert t1 <= 1.3 * tm, (t1, tm)
