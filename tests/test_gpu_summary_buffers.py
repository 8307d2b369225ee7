"""ssm_simulator_summary clears its six outputs wherever the caller keeps them.

Buffers that were allocated one by one may happen to lie directly behind one
another, and a clear must not treat such neighbours as one allocation; buffers
cut out of one block, in any order or with gaps, give the same counts.
"""

import ctypes

import numpy as np
import pytest
import torch

from ssms_b200 import _device as D
from ssms_b200 import _lib

pytestmark = pytest.mark.gpu

K, C, N, BINS = 32, 2, 5, (128, 256)  # 32 trials x 2 choices x 8 B: whole allocation granules
SIZES = [K * C, K * C, K, K, BINS[0] * C, BINS[1] * C]


def _call(at):
    rng = np.random.default_rng(2)
    rts = torch.from_numpy(rng.uniform(0.0, 3.0, N * K).astype(np.float32)).cuda()
    ch = torch.from_numpy(rng.choice(np.array([-1, 1], np.int32), N * K)).cuda()
    cv = torch.tensor([-1, 1], dtype=torch.int32, device="cuda")
    ea, eb = (torch.linspace(0, 3, n + 1, dtype=torch.float64, device="cuda") for n in BINS)
    _lib.check(_lib.lib().ssm_simulator_summary(
        D.ptr(rts), D.ptr(ch), N, K, D.ptr(cv), C, D.ptr(ea), BINS[0], D.ptr(eb), BINS[1], *at, D.stream_ptr()))
    torch.cuda.synchronize()


def _want():
    outs = [torch.full((n,), -1, dtype=torch.int64, device="cuda") for n in SIZES]
    _call([D.ptr(o) for o in outs])
    assert int(outs[0].sum()) == N * K
    return [o.cpu().numpy() for o in outs]


def test_adjacent_allocations(cuda):
    want = _want()
    rt = ctypes.CDLL("libcudart.so.12")  # the one torch has loaded
    rt.cudaMalloc.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t]
    rt.cudaFree.argtypes = [ctypes.c_void_p]
    rt.cudaMemcpy.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int]
    mine = []
    try:
        def one(nbytes):
            p = ctypes.c_void_p()
            assert rt.cudaMalloc(ctypes.byref(p), nbytes) == 0
            mine.append(p.value)
            return p.value

        # neighbours among single allocations: choice_counts followed by kept_counts
        step = 8 * SIZES[0]
        for _ in range(400):
            one(step)
        have = set(mine)
        first = next((p for p in sorted(mine) if p + step in have), None)
        if first is None:
            pytest.skip("the allocator placed no two buffers side by side")
        at = [first, first + step] + [one(8 * n) for n in SIZES[2:]]
        _call(at)
        for p, n, w in zip(at, SIZES, want):
            got = np.empty(n, np.int64)
            assert rt.cudaMemcpy(got.ctypes.data, p, 8 * n, 2) == 0
            np.testing.assert_array_equal(got, w)
    finally:
        for p in mine:
            rt.cudaFree(p)


@pytest.mark.parametrize("order", [(0, 1, 2, 3, 4, 5), (5, 3, 1, 0, 2, 4)])
@pytest.mark.parametrize("gap", [0, 3])
def test_one_block_in_any_order(cuda, order, gap):
    want = _want()
    block = torch.full((sum(SIZES) + 7 * gap,), -7, dtype=torch.int64, device="cuda")
    start, at = {}, gap
    for i in order:
        start[i] = at
        at += SIZES[i] + gap
    _call([D.ptr(block) + 8 * start[i] for i in range(6)])
    got = block.cpu().numpy()
    used = np.zeros(got.size, bool)
    for i, w in enumerate(want):
        np.testing.assert_array_equal(got[start[i]:start[i] + SIZES[i]], w)
        used[start[i]:start[i] + SIZES[i]] = True
    assert np.all(got[~used] == -7)
