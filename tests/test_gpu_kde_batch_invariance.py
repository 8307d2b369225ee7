"""A set's fit has the same bits in whatever call it is made.

How many blocks share a set depends on the number of sets in the call and on the
GPU; where the set begins in the arrays moves its loads against 16-byte
boundaries.  Neither may reach the results: points, bandwidths and proportions of
a set are those of a call with that set alone, bit for bit.
"""

import numpy as np
import pytest
import torch

from ssms_b200 import kde as gk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("displaced", [False, True])
@pytest.mark.parametrize("choices", [(-1, 1), (0, 1, 2), (0, 1, 2, 3, 4, 5)])
def test_one_set_alone_and_among_others(cuda, choices, displaced):
    rng = np.random.default_rng(len(choices))
    n = 5003
    rts = (0.3 + np.exp(rng.normal(0.0, 0.6, n))).astype(np.float32)
    rts[rng.uniform(size=n) < 0.03] = -999.0
    ch = rng.choice(np.asarray(choices, np.int32), n)

    def fit(before, n_sets):
        """The set at position 1, behind a set of `before` samples, among n_sets."""
        sizes = [before, n] + [257] * (n_sets - 2)
        total = int(np.sum(sizes))
        r, c = np.full(total, 0.7, np.float32), np.full(total, choices[0], np.int32)
        r[before:before + n], c[before:before + n] = rts, ch
        kb = gk.KdeBatch(torch.from_numpy(r), torch.from_numpy(c), np.concatenate([[0], np.cumsum(sizes)]),
                         list(choices), displace=np.full(n_sets, 0.25) if displaced else None)
        k = len(choices)
        po = kb.point_offsets.cpu().numpy()
        return (kb.points[int(po[k]):int(po[2 * k])].cpu(), kb.bandwidth[k:2 * k].cpu(), kb.log_norm[k:2 * k].cpu(),
                kb.proportion[k:2 * k].cpu())

    want = fit(0, 2)
    for before in (0, 1, 2, 3):
        for n_sets in (2, 80, 160, 400, 800):
            for got, exp in zip(fit(before, n_sets), want):
                assert torch.equal(got, exp), (before, n_sets)
