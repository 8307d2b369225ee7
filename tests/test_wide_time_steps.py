"""The closed form of the float32 time accumulator that walks on several lanes use.

TimeSteps (csrc/sim_wide.cu) takes an accumulator t = dt + dt + ... (n additions,
each rounded) and gives its value after m more additions without making them.  Its
argument needs n even, which every block start is.  The form is restated here in
numpy's float32 and compared with the additions for time steps whose additions become
ties at some point, for which an odd start would be wrong.
"""

import numpy as np

BLOCK = 144  # additions of a block: 18 steps for each of 8 lanes


def _accumulator(dt, n):
    return np.add.accumulate(np.concatenate([[np.float32(0)], np.full(n, dt, np.float32)]), dtype=np.float32)


def _off(dt, n=30_000):
    """By start 0 .. n - BLOCK: whether the form, where it is taken, misses an addition."""
    t = _accumulator(dt, n)
    t0, nxt = t[:-BLOCK], t[1:n - BLOCK + 2]
    inc = (nxt + dt).astype(np.float32) - nxt
    m = np.arange(1, BLOCK + 1)
    # fmaf: one rounding of a product and sum that float64 holds exactly
    form = (nxt.astype(np.float64)[:, None] + (m - 1) * inc.astype(np.float64)[:, None]).astype(np.float32)
    want = np.lib.stride_tricks.sliding_window_view(t, BLOCK + 1)[:, 1:]
    same_binade = np.frexp(nxt)[1] == np.frexp(form[:, -1])[1]
    return (form != want).any(axis=1) & same_binade & (t0 < 65536 * dt)


def test_even_starts_are_exact_and_odd_ones_need_not_be():
    rng = np.random.default_rng(5)
    odd_starts_off = 0
    for bits in (9, 10, 11, 12, 13, 14, 15, 15, 24, 24):
        odd = int(rng.integers(1 << (bits - 1), 1 << bits)) | 1
        dt = np.float32(odd * 2.0 ** (-10 - bits))  # between 2^-11 and 2^-10
        off = _off(dt)
        assert not off[0::2].any(), (bits, odd)
        odd_starts_off += int(off[1::2].sum())
    assert not _off(np.float32(0.001))[0::2].any()
    assert odd_starts_off > 0  # what the even starts keep out
