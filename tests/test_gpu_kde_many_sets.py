"""Calls of more than 2^28 sets, as many as a grid has blocks for (2^31 - 1).

All sets but the last are empty: the last one's counts, proportion and histogram
show that every set was reached.
"""

import pytest
import torch

from ssms_b200 import _device as D
from ssms_b200 import _lib

pytestmark = pytest.mark.gpu

S = (1 << 28) + 3
RTS, CHOICES = [0.5, 1.5, -999.0, 0.7, 0.2], [1, 1, 1, -1, 1]


@pytest.fixture
def sets(cuda):
    if torch.cuda.mem_get_info()[0] < 32 << 30:
        pytest.skip("needs 20 GB of device memory")
    soff = torch.zeros(S + 1, dtype=torch.int64, device="cuda")
    soff[-1] = len(RTS)
    yield (torch.tensor(RTS, device="cuda"), torch.tensor(CHOICES, dtype=torch.int32, device="cuda"), soff,
           torch.tensor([1], dtype=torch.int32, device="cuda"))
    del soff
    torch.cuda.empty_cache()


def _new(dtype, n):
    return torch.full((n,), -5, dtype=dtype, device="cuda")


def test_fit(sets):
    rts, choices, soff, cv = sets
    call, nval, poff = (_new(torch.int64, n) for n in (S, S, S + 1))
    h, ln, prop = (_new(torch.float64, S) for _ in range(3))
    points = torch.empty(len(RTS), device="cuda")
    _lib.check(_lib.lib().ssm_kde_fit(
        D.ptr(rts), D.ptr(choices), S, D.ptr(soff), D.ptr(cv), 1, None, None, D.ptr(call), D.ptr(nval), D.ptr(poff),
        D.ptr(points), D.ptr(h), D.ptr(ln), D.ptr(prop), D.stream_ptr()))
    assert int(call[-1]) == 4 and int(call[:-1].abs().sum()) == 0
    assert int(nval[-1]) == 3 and int(nval[:-1].abs().sum()) == 0
    assert int(poff[-1]) == 3 and int(poff[:-1].abs().sum()) == 0
    assert float(prop[-1]) == 0.8 and float(prop[:-1].abs().sum()) == 0.0
    assert float(h[-1]) > 0.0 and bool((h[:-1] == -1.0).all())


def test_summary(sets):
    rts, choices, soff, cv = sets
    counts, nogo, omit = (_new(torch.int64, S) for _ in range(3))
    ha, hb = _new(torch.float32, S), _new(torch.float32, 2 * S)
    _lib.check(_lib.lib().ssm_set_summary(
        D.ptr(rts), D.ptr(choices), S, D.ptr(soff), D.ptr(cv), 1, 2.0, D.ptr(counts), D.ptr(nogo), D.ptr(omit),
        1, D.ptr(ha), 2, D.ptr(hb), D.stream_ptr()))
    assert int(counts[-1]) == 4 and int(counts[:-1].abs().sum()) == 0
    assert int(nogo[-1]) == 2 and int(nogo[:-1].abs().sum()) == 0
    assert int(omit.abs().sum()) == 0
    assert hb[-2:].tolist() == [2.0, 1.0] and float(hb[:-2].abs().double().sum()) == 0.0
    assert float(ha[-1]) == 3.0 and float(ha[:-1].abs().double().sum()) == 0.0
