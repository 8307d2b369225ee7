"""Walks on several lanes against walks that never leave their one lane.

A workspace of the size that the entry points require, without the room for walks
that are handed over, keeps a launch of one lane per walk on one lane to its end.
Launches that hand their last walks over and launches of 8, 16 or 32 lanes per walk
must give the same bits: rts, choices, step counts and the recorded trajectory, for
every model and in-register bound, in both layouts.  Many walks here end at a time
limit.  Two of the time steps are odd multiples of half an ulp of the float32 time
accumulator, from 1 s and from 2 s on, where every addition is a tie.
"""

import numpy as np
import pytest
import torch

from ssms_b200 import _device as D
from ssms_b200 import _lib
from ssms_b200 import device as dev

pytestmark = pytest.mark.gpu

K, MAX_T = 24, 3.0
DTS = [0.001, 15979 / 2**24, 7989 / 2**23]
GAUSSIAN = ["ddm_flexbound", "ddm_sdv", "full_ddm", "ornstein_uhlenbeck"]
KINDS = [_lib.BOUND_CONSTANT, _lib.BOUND_LINEAR, _lib.BOUND_WEIBULL]
CASES = [(m, k) for m in [*GAUSSIAN, "levy_flexbound", "ddm_flex"] for k in KINDS] + [("ddm", _lib.BOUND_CONSTANT)]
f32 = lambda x: np.asarray(x, np.float32)  # noqa: E731


def _inputs(model, kind):
    rng = np.random.default_rng(47)
    u = lambda lo, hi: f32(rng.uniform(lo, hi, K))  # noqa: E731
    kw = {"v": u(-0.6, 0.6), "a": u(1.2, 2.6), "z": u(0.4, 0.6), "t": u(0.0, 0.5), "s": f32(np.ones(K)),
          "deadline": f32(np.where(np.arange(K) % 3 == 0, 1.8, 999.0)), "bound_kind": kind}
    if kind == _lib.BOUND_LINEAR:
        kw["bound_p1"] = -u(0.02, 0.2)
    if kind == _lib.BOUND_WEIBULL:
        kw["bound_p1"], kw["bound_p2"] = u(1, 3), u(4, 8)
    extra = {"levy_flexbound": {"alpha": u(1.5, 2.0)}, "ddm_sdv": {"sv": u(0.1, 0.5)},
             "full_ddm": {"sv": u(0.1, 0.5), "sz": u(0.01, 0.1), "st": u(0.01, 0.2)},
             "ornstein_uhlenbeck": {"g": u(-0.3, 0.6)},
             "ddm_flex": {"drift_table": f32(rng.uniform(-0.8, 0.8, (K, 3201)))}}
    kw.update(extra.get(model, {}))
    return kw


def _runner(model, kind, dt):
    kw = _inputs(model, kind)

    def run(lanes, **more):
        """The outputs' bits, and how many walks were handed over."""
        shape = more.pop("shape", (0, 0, 0))
        out = dev.simulate_single(model, n_trials=K, max_t=MAX_T, delta_t=dt, seed=77, smooth_unif=True,
                                  want_steps=True, launch=D.launch_opts(*shape, lanes_per_walk=lanes), **kw, **more)
        assert _lib.lib().ssm_check_status(D.ptr(out.workspace), D.stream_ptr()) == _lib.SSM_OK
        got = [out.rts.view(torch.int32), out.choices, out.steps]
        if out.traj is not None:
            got.append(out.traj.view(torch.int32))
        handed = int(out.workspace[:256].view(torch.int64)[2])
        return [x.cpu().numpy() for x in got], handed

    return run


@pytest.fixture
def required_workspace(monkeypatch):
    """Switch to the workspace without hand-over room, and back."""
    L = _lib.lib()
    full = L.ssm_ddm_workspace_bytes

    def use(small):
        monkeypatch.setattr(L, "ssm_ddm_workspace_bytes",
                            (lambda n: (256 + 64 * n + 255) // 256 * 256) if small else full)

    yield use


def _equal(got, want):
    for g, w, name in zip(got, want, ("rts", "choices", "steps", "trajectory")):
        np.testing.assert_array_equal(g, w, err_msg=name)


@pytest.mark.parametrize("dt", DTS)
@pytest.mark.parametrize("model,kind", CASES)
def test_reference_layout(cuda, required_workspace, model, kind, dt):
    run = _runner(model, kind, dt)
    n = 100 * torch.cuda.get_device_properties(0).multi_processor_count // K + 9  # enough for 8 lanes a walk
    required_workspace(True)
    want, handed = run(1, n_samples=n, traj_len=3400)
    assert handed == 0
    assert (want[2] > (MAX_T - 0.6) / dt).mean() > 0.01  # walks that reach their time limit
    required_workspace(False)
    for shape in ((0, 0, 0), (32, 1, 32)):
        got, handed = run(1, n_samples=n, traj_len=3400, shape=shape)
        assert handed > 0
        _equal(got, want)
    if model in ("levy_flexbound", "ddm_flex"):
        return
    for m, lanes in ((n, 8), (n // 2, 8), (n // 5, 8), (n // 5, 0), (n, 4), (n, 2)):
        _equal(run(lanes, n_samples=m, traj_len=3400)[0], [*(x[:m * K] for x in want[:3]), want[3]])


@pytest.mark.parametrize("dt", DTS)
@pytest.mark.parametrize("model,kind", CASES)
def test_ragged_layout(cuda, required_workspace, model, kind, dt):
    run = _runner(model, kind, dt)
    ns = np.random.default_rng(3).integers(1, 600, K)
    ns[[3, 17]] = 0
    offs = np.concatenate([[0], np.cumsum(ns)]).astype(np.int64)
    required_workspace(True)
    want, handed = run(1, sample_offsets=offs)
    assert handed == 0
    if model not in ("levy_flexbound", "ddm_flex"):
        _equal(run(4, sample_offsets=offs)[0], want)  # eight lanes where nothing can be handed over
    required_workspace(False)
    for shape in ((0, 0, 0), (32, 1, 32)):
        got, handed = run(1, sample_offsets=offs, shape=shape)
        assert handed > 0
        _equal(got, want)
    if model not in ("levy_flexbound", "ddm_flex"):
        for lanes in (8, 4, 2, 0):
            _equal(run(lanes, sample_offsets=offs)[0], want)
