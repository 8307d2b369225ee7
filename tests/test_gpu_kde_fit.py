"""The KDE fit's compaction and moments at the edges of its slices and chunks.

Every set is cut into one slice per CTA of its cluster and each slice into
chunks of 1 024 samples, four per thread; these sizes sit around those edges,
with unaligned and mutually misaligned inputs, one to many choices, and set
counts that take every cluster size.  Points must be the stable per-choice
compaction of float32 log-rts (the device logarithm is float64, so its float32
rounding agrees with numpy's to one ulp), counts exact; bandwidths follow from
the points in float64, where another summation order moves the last few of 52
bits (1e-12 relative allows n eps for the sizes here).
"""

import numpy as np
import pytest
import torch

from ssms_b200 import kde as gk

pytestmark = pytest.mark.gpu


def _check(sizes, choices, shift_r, shift_c, seed):
    rng = np.random.default_rng(seed)
    n = int(np.sum(sizes))
    rts = np.exp(rng.normal(0.0, 0.6, n)).astype(np.float32)
    rts[rng.uniform(size=n) < 0.05] = -999.0
    ch = rng.choice(np.asarray(list(choices) + [77], np.int32), n)  # 77 belongs to no group
    r = torch.zeros(n + 8, dtype=torch.float32, device="cuda")
    c = torch.zeros(n + 8, dtype=torch.int32, device="cuda")
    r[shift_r:shift_r + n] = torch.from_numpy(rts).cuda()
    c[shift_c:shift_c + n] = torch.from_numpy(ch).cuda()
    soff = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    kb = gk.KdeBatch(r[shift_r:shift_r + n], c[shift_c:shift_c + n], soff, list(choices))
    cv, poff = kb.choice_values, kb.point_offsets.cpu().numpy()
    pts, h, prop = (x.cpu().numpy() for x in (kb.points, kb.bandwidth, kb.proportion))
    call = kb.count_all.cpu().numpy()
    g = 0
    for s in range(len(sizes)):
        rs, cs = rts[soff[s]:soff[s + 1]], ch[soff[s]:soff[s + 1]]
        for v in cv:
            assert call[g] == np.sum(cs == v)
            want = np.log(rs[(cs == v) & (rs != -999.0)].astype(np.float64)).astype(np.float32)
            assert poff[g + 1] - poff[g] == want.size
            got = pts[poff[g]:poff[g + 1]]
            assert np.all(np.abs(got - want) <= np.spacing(np.abs(want)))
            if want.size == 0:
                assert h[g] == -1.0
            else:
                np.testing.assert_allclose(h[g], gk.bandwidth_silverman(got.astype(np.float64)), rtol=1e-12)
                assert prop[g] == np.sum(cs == v) / cs.size
            g += 1


@pytest.mark.parametrize("choices", [(-1, 1), (0, 1, 2), (0, 1, 2, 3), (0, 1, 2, 3, 4, 5, 6)])
@pytest.mark.parametrize("shift_r,shift_c", [(0, 0), (1, 1), (3, 2)])
def test_chunk_and_slice_edges(cuda, choices, shift_r, shift_c):
    _check([0, 1, 2, 3, 5, 31, 1023, 1024, 1025, 4097, 8191, 8192, 8193, 20011], choices, shift_r, shift_c, 1)


@pytest.mark.parametrize("n_sets", [1, 75, 150, 300, 700])
def test_cluster_sizes(cuda, n_sets):
    _check(list(100 + (np.arange(n_sets) * 37) % 200), (-1, 1), 0, 0, n_sets)


def test_evaluation_unit_and_tile_edges(cuda):
    """Query counts around a row (32), a unit (512) and several units, point
    counts around a staged tile (512) and the 32-term groups, empty groups on
    either side: against the float64 sum over the fitted points, with the
    tolerance of the KDE evaluation (1e-5 absolute plus 2e-6 relative)."""
    rng = np.random.default_rng(3)
    n_pts = [0, 1, 31, 32, 33, 511, 512, 513, 1025, 5000]
    n_q = [0, 1, 31, 32, 33, 511, 512, 513, 1024, 1537]
    pairs = [(p, q) for p in n_pts for q in n_q]
    sizes = np.array([p for p, _ in pairs])
    rts = np.exp(rng.normal(0.0, 0.5, int(sizes.sum()))).astype(np.float32)
    soff = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    kb = gk.KdeBatch(torch.from_numpy(rts), torch.ones(rts.size, dtype=torch.int32), soff, [1])
    qoff = np.concatenate([[0], np.cumsum([q for _, q in pairs])]).astype(np.int64)
    q = np.exp(rng.normal(0.0, 0.8, int(qoff[-1])))
    q[::97] = 0.0  # not after the start: the floor
    ll = kb.evaluate(qoff, torch.from_numpy(q), max_t=20.0).cpu().numpy()
    pts, h = kb.points.cpu().numpy().astype(np.float64), kb.bandwidth.cpu().numpy()
    for g, (p, m) in enumerate(pairs):
        got, qq = ll[qoff[g]:qoff[g + 1]], q[qoff[g]:qoff[g + 1]]
        if p == 0:
            with np.errstate(divide="ignore"):
                np.testing.assert_array_equal(got, np.full(m, -np.log(np.float64(0.0) * 20.0)))
            continue
        lq = np.log(np.maximum(qq, 1e-4))
        d = (lq[:, None] - pts[None, soff[g]:soff[g + 1]]) / h[g]
        with np.errstate(divide="ignore"):
            want = np.log(np.exp(-0.5 * d * d).sum(axis=1) / (p * h[g] * np.sqrt(2 * np.pi))) - lq
        want = np.where((qq > 0) & (want > -66.774), want, -66.774)
        floor = (got == -66.774) | (want == -66.774)
        np.testing.assert_allclose(got[~floor], want[~floor], rtol=2e-6, atol=1e-5)
        assert np.all(np.abs(got - want)[floor] < 1e-3)
