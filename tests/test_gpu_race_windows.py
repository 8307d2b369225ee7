"""Race, LCA and racing diffusion walks do not depend on the way they are run.

With up to four accumulators a walk goes through windows of steps: without a test
each where the window cannot end it, step by step where it may; on its own lane
in a full launch, on draws shared by the warp's lanes at a launch's end and in a
small one.  A walk depends on (seed, trial, sample) alone, so all of these must
agree bit for bit in rts, choices and step counts, and with the trajectory
recorder, which takes every step with its tests.
"""

import numpy as np
import pytest
import torch

from ssms_b200 import _device as D
from ssms_b200 import _lib
from ssms_b200 import device as dev

pytestmark = pytest.mark.gpu

K = 6
f32 = lambda x: np.asarray(x, np.float32)  # noqa: E731
KINDS = [_lib.BOUND_TABLE, _lib.BOUND_CONSTANT, _lib.BOUND_LINEAR, _lib.BOUND_WEIBULL]
CASES = [(f, n, k) for f in ("race_model", "lca") for n in (2, 3, 4) for k in KINDS] + [("rdm", n, None) for n in (2, 3, 4)]


def _run(family, n_acc, kind, n_samples, delta_t=0.001, max_t=1.2, high=1.0, **more):
    rng = np.random.default_rng(17)
    u = lambda lo, hi, *sh: f32(rng.uniform(lo, hi, (K, *sh)))  # noqa: E731
    kw = {"v": u(0.0, 2.0, n_acc), "t": u(0.0, 0.5), "n_trials": K, "n_samples": n_samples, "max_t": max_t,
          # deadlines inside a window, past max_t, and one that has passed before the first step
          "deadline": f32([0.731, 999.0, 1.0, 999.0, 0.2, 999.0]), "delta_t": delta_t, "seed": 91,
          "smooth_unif": True, "want_steps": True, **more}
    if family == "rdm":
        return dev.simulate_rdm(b=high * u(0.5, 1.5), A=u(0.1, 0.4), s=f32(np.ones(K)), **kw)
    kw.update(z=u(0.0, 0.5, n_acc), s=f32(np.ones((K, n_acc))), a=high * u(0.6, 1.6), bound_kind=kind)
    if kind == _lib.BOUND_LINEAR:
        kw["bound_p1"] = f32([-0.5, 0.4, -2.0, 0.0, -0.1, -1.0])
    if kind == _lib.BOUND_WEIBULL:
        kw["bound_p1"], kw["bound_p2"] = u(0.5, 3), u(0.5, 4)
    if kind == _lib.BOUND_TABLE:
        kw["bound_table"] = kw["a"][:, None] * np.linspace(1, 0.2, 1201, dtype=np.float32)[None]
    if family == "lca":
        kw.update(g=u(-1.0, 1.0), b=u(-1.0, 1.0))
    return dev.simulate_race(family, **kw)


def _bits(o):
    assert _lib.lib().ssm_check_status(D.ptr(o.workspace), D.stream_ptr()) == _lib.SSM_OK
    return [o.rts.view(torch.int32).cpu().numpy(), o.choices.cpu().numpy(), o.steps.cpu().numpy()]


@pytest.mark.parametrize("family,n_acc,kind", CASES)
def test_launch_sizes_and_shapes_agree(cuda, family, n_acc, kind):
    one = D.launch_opts(32, 1, 32)  # 148 warps of one block per SM: many walks each
    want = [x.reshape(3000, K) for x in _bits(_run(family, n_acc, kind, 3000, launch=one))]
    assert len(np.unique(want[2])) > 20
    for n, shape in ((1, (256, 0, 32, 0)), (40, (256, 0, 32, 0)), (90, (32, 1, 32, 0)), (700, (32, 1, 32, 1)),
                     (3000, (256, 0, 256, 32)), (3000, (64, 2, 64, 4))):
        got = _bits(_run(family, n_acc, kind, n, launch=D.launch_opts(*shape[:3], refill_min=shape[3])))
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g.reshape(n, K), w[:n])


@pytest.mark.parametrize("family,n_acc,kind", CASES)
@pytest.mark.parametrize("first", [{}, {"max_t": 0.0}, {"delta_t": 1e-5, "max_t": 0.9, "high": 50.0}])
def test_recorded_path_ends_where_the_walk_does(cuda, family, n_acc, kind, first):
    """{}: ends at a bound or its time; no step; more than 65 536 steps (the time limit)."""
    o = _run(family, n_acc, kind, 1, traj_len=100_000 * n_acc, **first)
    steps, path = int(o.steps[0]), o.traj.cpu().numpy().reshape(-1, n_acc)
    taken = int((path != -999.0).all(axis=1).sum()) - 1
    # racing diffusion's last step (the one that reaches the bound) is not counted or recorded
    assert taken == steps
    if steps and family != "rdm":
        assert int(path[steps].argmax()) == int(o.choices[0])
