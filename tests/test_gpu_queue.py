"""The work queue's restart paths give every walk the same result.

A walk depends on (seed, trial, sample) alone, so one parameter set per trial,
simulated (a) in the reference layout, (b) ragged in index order, (c) ragged in
a given order, with trials of no, one and many samples, and under launch shapes
that take the queue's different routes (restarts inside the warp's last trial,
across trials, claims that run out, one to many walks per warp), must agree bit
for bit: rts, choices and step counts, for every model and boundary form.  The
rts that a launch leaves to its finishing kernel are part of that.
"""

import numpy as np
import pytest
import torch

from ssms_b200 import _device as D
from ssms_b200 import _lib
from ssms_b200 import device as dev
from ssms_b200.batch import with_order

pytestmark = pytest.mark.gpu

NS = np.array([40, 0, 129, 1, 1, 1, 64, 0, 700, 33, 2, 257])
K = NS.size
f32 = lambda x: np.asarray(x, np.float32)  # noqa: E731


def _inputs(model, kind):
    rng = np.random.default_rng(31)
    u = lambda lo, hi: f32(rng.uniform(lo, hi, K))  # noqa: E731
    kw = {"v": u(-2, 2), "a": u(0.4, 1.5), "z": u(0.2, 0.8), "t": u(0.0, 1.0), "s": f32(np.ones(K)),
          "deadline": f32(np.where(np.arange(K) % 3 == 0, 1.5, 999.0)), "bound_kind": kind}
    if kind == _lib.BOUND_LINEAR:
        kw["bound_p1"] = -u(0.1, 0.8)
    if kind == _lib.BOUND_WEIBULL:
        kw["bound_p1"], kw["bound_p2"] = u(0.5, 3), u(0.5, 4)
    if kind == _lib.BOUND_TABLE:
        kw["bound_table"] = kw["a"][:, None] * np.linspace(1, 0.2, 3001, dtype=np.float32)[None]
    extra = {"levy_flexbound": {"alpha": u(1.0, 2.0)}, "ddm_sdv": {"sv": u(0.1, 1)},
             "full_ddm": {"sv": u(0.1, 1), "sz": u(0.01, 0.2), "st": u(0.01, 0.2)},
             "ornstein_uhlenbeck": {"g": u(-1, 1)},
             "ddm_flex": {"drift_table": f32(rng.uniform(-2, 2, (K, 3001)))}}
    kw.update(extra.get(model, {}))
    return kw


def _bits(out):
    return [out.rts.view(torch.int32).cpu().numpy(), out.choices.cpu().numpy(), out.steps.cpu().numpy()]


MODELS = ["ddm_flexbound", "levy_flexbound", "ddm_sdv", "full_ddm", "ornstein_uhlenbeck", "ddm_flex"]
KINDS = [_lib.BOUND_TABLE, _lib.BOUND_CONSTANT, _lib.BOUND_LINEAR, _lib.BOUND_WEIBULL]
CASES = [(m, k) for m in MODELS for k in KINDS] + [("ddm", _lib.BOUND_CONSTANT)]


@pytest.mark.parametrize("model,kind", CASES)
def test_layouts_orders_and_shapes_agree(cuda, model, kind):
    kw = _inputs(model, kind)
    n_max = int(NS.max())
    run = lambda **more: dev.simulate_single(model, n_trials=K, max_t=3.0, seed=77, smooth_unif=True,  # noqa: E731
                                             want_steps=True, **kw, **more)
    ref = _bits(run(n_samples=n_max, launch=D.launch_opts(lanes_per_walk=1)))
    full = [x.reshape(n_max, K) for x in ref]
    want = [np.concatenate([x[:NS[k], k] for k in range(K)]) for x in full]
    offs = np.concatenate([[0], np.cumsum(NS)]).astype(np.int64)
    order = np.random.default_rng(3).permutation(K).astype(np.int32)
    qoff = np.concatenate([[0], np.cumsum(NS[order])]).astype(np.int64)
    ot, qt = torch.from_numpy(order).cuda(), torch.from_numpy(qoff).cuda()
    wide = [1] if model in ("levy_flexbound", "ddm_flex") or kind == _lib.BOUND_TABLE else [1, 2, 4, 8]
    for w in wide:
        for shape in ((32, 1, 32, 1), (64, 1, 256, 2), (256, 0, 64, 32)):
            lo = D.launch_opts(*shape[:3], refill_min=shape[3], lanes_per_walk=w)
            for launch in (lo, with_order(lo, ot, qt)):
                out = run(sample_offsets=offs, launch=launch)
                assert _lib.lib().ssm_check_status(D.ptr(out.workspace), D.stream_ptr()) == _lib.SSM_OK
                for got, exp in zip(_bits(out), want):
                    np.testing.assert_array_equal(got, exp)


@pytest.mark.parametrize("model,kind", [c for c in CASES if c[0] not in ("levy_flexbound", "ddm_flex")
                                        and c[1] != _lib.BOUND_TABLE])
def test_group_widths_agree(cuda, model, kind):
    """A launch of known size takes 32, 16 or 8 lanes per walk (up to 24, 96 and more
    walks per SM): the walks are those of one lane each."""
    kw = _inputs(model, kind)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    run = lambda n, w: _bits(dev.simulate_single(model, n_trials=K, n_samples=n, max_t=3.0, seed=77,  # noqa: E731
                                                 smooth_unif=True, want_steps=True, launch=D.launch_opts(lanes_per_walk=w),
                                                 **kw))
    want = run(100 * sms // K + 9, 1)
    for walks in (1, 24 * sms, 24 * sms + 12, 96 * sms, 96 * sms + 24):
        n = max(1, walks // K)
        for w in (0, 8):
            for got, exp in zip(run(n, w), want):
                np.testing.assert_array_equal(got, exp[:n * K])


@pytest.mark.parametrize("model,kind", CASES)
def test_injected_noise_agrees_across_layouts(cuda, model, kind):
    kw = _inputs(model, kind)
    rng = np.random.default_rng(8)
    ns = np.minimum(NS, 70)
    offs = np.concatenate([[0], np.cumsum(ns)]).astype(np.int64)
    n_max, row = int(ns.max()), 3003
    rows = torch.randn(n_max * K, row, device="cuda", generator=torch.Generator("cuda").manual_seed(4))
    per = 3 if model == "full_ddm" else 1
    unif = f32(rng.uniform(0, 1, (n_max * K, per)))
    run = lambda **more: dev.simulate_single(model, n_trials=K, max_t=3.0, smooth_unif=True, want_steps=True,  # noqa: E731
                                             **kw, **more)
    ref = _bits(run(n_samples=n_max, noise_rows=rows, noise_unif=unif.reshape(-1)))
    pick = np.concatenate([np.arange(ns[k]) * K + k for k in range(K)]).astype(np.int64)
    rows_r, unif_r = rows[torch.from_numpy(pick).cuda()].contiguous(), unif[pick].reshape(-1)
    for shape in ((32, 1, 32, 1), (128, 0, 256, 2)):
        out = run(sample_offsets=offs, noise_rows=rows_r, noise_unif=unif_r,
                  launch=D.launch_opts(*shape[:3], refill_min=shape[3]))
        for got, exp in zip(_bits(out), ref):
            np.testing.assert_array_equal(got, exp[pick])
