"""Counts of a set with more than 2^32 samples.

With several hundred sets in a call one block counts a whole set, so its counters
have to hold all of the set's samples: the fit's counts, the summary's counts and
the histogram bin that takes them all.  The samples are one int32 pattern that both
arrays share: as an rt it is -999 (an omission) or a positive denormal (the first
bin), as a choice the one that is counted.
"""

import numpy as np
import pytest
import torch

from ssms_b200 import _device as D
from ssms_b200 import _lib

pytestmark = pytest.mark.gpu

N = (1 << 32) + 5


@pytest.fixture(scope="module")
def pattern(cuda):
    if torch.cuda.mem_get_info()[0] < 24 << 30:
        pytest.skip("needs 17 GB of device memory for one array of samples")
    x = torch.empty(N, dtype=torch.int32, device="cuda")
    yield x
    del x
    torch.cuda.empty_cache()


def _sets(first):
    n_sets = 4 * torch.cuda.get_device_properties(0).multi_processor_count + 8  # one block per set
    soff = torch.full((n_sets + 1,), first, dtype=torch.int64, device="cuda")
    soff[0] = 0
    return n_sets, soff


def test_fit_counts(pattern):
    bits = int(np.array(-999.0, np.float32).view(np.int32))
    pattern.fill_(bits)
    S, soff = _sets(N)
    cv = torch.tensor([bits, 7], dtype=torch.int32, device="cuda")
    i64 = lambda n: torch.empty(n, dtype=torch.int64, device="cuda")  # noqa: E731
    f64 = lambda n: torch.empty(n, dtype=torch.float64, device="cuda")  # noqa: E731
    call, nval, poff, h, ln, prop = i64(2 * S), i64(2 * S), i64(2 * S + 1), f64(2 * S), f64(2 * S), f64(2 * S)
    points = torch.empty(1, device="cuda")
    _lib.check(_lib.lib().ssm_kde_fit(
        D.ptr(pattern), D.ptr(pattern), S, D.ptr(soff), D.ptr(cv), 2, None, None, D.ptr(call), D.ptr(nval), D.ptr(poff),
        D.ptr(points), D.ptr(h), D.ptr(ln), D.ptr(prop), D.stream_ptr()))
    assert call[:4].tolist() == [N, 0, 0, 0]
    assert int(nval.abs().sum()) == 0 and int(poff[-1]) == 0
    assert prop[:2].tolist() == [1.0, 0.0]


@pytest.mark.parametrize("bins", [(128, 256), (100, 256)])  # the first from the second by pairs, and on its own
def test_summary_counts(pattern, bins):
    pattern.fill_(3)  # 4e-45 as a float
    S, soff = _sets(N)
    cv = torch.tensor([-1, 3], dtype=torch.int32, device="cuda")
    i64 = lambda n: torch.empty(n, dtype=torch.int64, device="cuda")  # noqa: E731
    counts, nogo, omit = i64(2 * S), i64(S), i64(S)
    ha, hb = (torch.empty(S * b * 2, device="cuda") for b in bins)
    _lib.check(_lib.lib().ssm_set_summary(
        D.ptr(pattern), D.ptr(pattern), S, D.ptr(soff), D.ptr(cv), 2, 20.0, D.ptr(counts), D.ptr(nogo), D.ptr(omit),
        bins[0], D.ptr(ha), bins[1], D.ptr(hb), D.stream_ptr()))
    assert counts[:4].tolist() == [0, N, 0, 0]
    assert int(nogo.sum()) == 0 and int(omit.sum()) == 0
    for hist, b in ((ha, bins[0]), (hb, bins[1])):
        hist = hist.reshape(S, b, 2)
        assert float(hist[0, 0, 1]) == float(np.float32(N))
        assert float(hist.double().sum()) == float(np.float32(N))
