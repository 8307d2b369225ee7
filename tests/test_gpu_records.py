"""Record shuffle and per-set summaries at their edges.

The shuffle's rounds must give the permutation of the sequential Fisher-Yates
loop over the same Philox draws, and the summary the counts and histograms of
numpy, exactly.
"""

import numpy as np
import pytest
import torch

from ssms_b200 import _device as D
from ssms_b200 import _lib

pytestmark = pytest.mark.gpu


def _philox(c, seed):
    """Philox4x32-10 (Salmon, Moraes, Dror & Shaw, SC'11) over counter arrays [4, n]."""
    c = [np.asarray(x, np.uint64) for x in c]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    m = np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


@pytest.mark.parametrize("M", [1, 2, 3, 255, 256, 257, 1000, 4097, 12288])
def test_shuffle_is_the_sequential_one(cuda, M):
    S, seed = 3, 0x1234567890ABCDEF
    q = torch.arange(S * M, dtype=torch.float64, device="cuda")
    qoff = torch.arange(0, S * M + 1, M, dtype=torch.int64, device="cuda")
    th = torch.zeros(S, 1, device="cuda")
    cv = torch.ones(1, dtype=torch.int32, device="cuda")
    out = torch.empty(S * M, 4, device="cuda")
    _lib.check(_lib.lib().ssm_kde_records(D.ptr(th), 1, S, 1, D.ptr(cv), D.ptr(qoff), D.ptr(q), D.ptr(q), 0, M, 0.0,
                                          seed, D.ptr(out), D.stream_ptr()))
    got = out[:, 1].cpu().numpy().reshape(S, M)
    for s in range(S):
        i = np.arange(M, dtype=np.uint64)
        w = _philox([i, np.full(M, s), np.zeros(M), np.full(M, 9)], seed)
        u = ((w[0] >> np.uint64(5)).astype(np.float64) * 67108864.0 + (w[1] >> np.uint64(6)).astype(np.float64)) / 2.0**53
        j = np.minimum((u * (np.arange(M) + 1.0)).astype(np.int64), np.arange(M))
        perm = np.arange(M)
        for k in range(M - 1, 0, -1):
            perm[k], perm[j[k]] = perm[j[k]], perm[k]
        want = np.empty(M)
        want[perm] = s * M + np.arange(M)
        np.testing.assert_array_equal(got[s], want)


@pytest.mark.parametrize("choices", [(-1, 1), (0, 1, 2), (0, 1, 2, 3, 4, 5)])
@pytest.mark.parametrize("bins", [(128, 256), (100, 256)])
@pytest.mark.parametrize("max_t", [20.0, 3.3])
def test_summary_matches_numpy(cuda, choices, bins, max_t):
    rng = np.random.default_rng(5)
    max_t = float(np.float32(max_t))
    sizes = [0, 1, 5, 1023, 4100, 30011]
    n = sum(sizes)
    rts = rng.uniform(0, 1.1 * max_t, n).astype(np.float32)
    edge = rng.uniform(size=n) < 0.3  # values on bin edges, and the closing edge
    rts[edge] = (np.linspace(0, max_t, bins[1] + 1)[rng.integers(0, bins[1] + 1, int(edge.sum()))]).astype(np.float32)
    rts[rng.uniform(size=n) < 0.05] = -999.0
    ch = rng.choice(np.asarray(list(choices) + [-999, 55], np.int32), n)
    soff = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    S, C = len(sizes), len(choices)
    r, c, o = torch.from_numpy(rts).cuda(), torch.from_numpy(ch).cuda(), torch.from_numpy(soff).cuda()
    cv = torch.as_tensor(np.asarray(choices, np.int32)).cuda()
    i64 = lambda k: torch.full((k,), -7, dtype=torch.int64, device="cuda")  # noqa: E731
    cnt, nogo, omit = i64(S * C), i64(S), i64(S)
    ha, hb = (torch.full((S, b, C), -7.0, device="cuda") for b in bins)
    _lib.check(_lib.lib().ssm_set_summary(D.ptr(r), D.ptr(c), S, D.ptr(o), D.ptr(cv), C, max_t, D.ptr(cnt),
                                          D.ptr(nogo), D.ptr(omit), bins[0], D.ptr(ha), bins[1], D.ptr(hb),
                                          D.stream_ptr()))
    cnt = cnt.cpu().numpy().reshape(S, C)
    for s in range(S):
        rs, cs = rts[soff[s]:soff[s + 1]], ch[soff[s]:soff[s + 1]]
        assert nogo[s].item() == np.sum((cs != max(choices)) | (rs == -999.0))
        assert omit[s].item() == np.sum(cs == -999)
        for k, v in enumerate(choices):
            assert cnt[s, k] == np.sum(cs == v)
            x = rs[(cs == v) & (rs != -999.0)].astype(np.float64)
            for h, b in ((ha, bins[0]), (hb, bins[1])):
                want, _ = np.histogram(x, bins=np.linspace(0, max_t, b + 1))
                np.testing.assert_array_equal(h[s, :, k].cpu().numpy(), want)
