"""The step adjoint at the sizes where its kernels change their lanes per slot (a warp, 16, 4).

Reverse-mode gradients of a random linear functional of the final state against central
differences of the FP64 forward on the same GPU, to the adjoint tests' 1e-3. Three steps of 0.05
m/s move a particle by 2e-3 of the spacing, and the jitter leaves neighbours 0.98 spacings apart,
so no pair comes under the collision distance of 0.9: the rollout is smooth in the velocities and
a relative step of 1e-6 puts truncation and rounding of the differences under 1e-6.
"""
from __future__ import annotations

import math

import numpy as np
import pytest

from mps_cuda_b200 import SceneDesc, configs
from mps_cuda_b200 import _lib as L
from mps_cuda_b200.adjoint import RolloutProblem

pytestmark = pytest.mark.gpu


def _dot(a, b):
    return math.fsum((np.asarray(a) * np.asarray(b)).ravel())


@pytest.mark.parametrize("block,tank,steps,every", [
    ((1, 1, 2), (5, 4, 6), 3, 3),
    ((3, 7, 11), (9, 7, 13), 5, 2),       # three segments, the last one short
    ((25, 8, 25), (31, 9, 27), 3, 3),     # 5000: the last size of a warp each
    ((23, 17, 13), (40, 17, 15), 3, 3),   # 5083: 16 lanes each
    ((46, 46, 47), (60, 46, 50), 2, 2),   # 99 452: 4 lanes each
])
def test_gradient_at_the_lines_of_the_lane_rule(block, tank, steps, every):
    l0 = 0.02
    pr = RolloutProblem(SceneDesc(l0, tuple(t * l0 for t in tank), block, seed=5, vel_sigma=0.05,
                                  vel_seed=2), dt=2e-4, steps=steps, every=every)
    n, f = pr.typ.shape[0], pr.fluid
    rng = np.random.default_rng(7)
    a, b, d = (rng.standard_normal((3, f.size)) for _ in range(3))
    lam_pos, lam_vel = np.zeros((3, n)), np.zeros((3, n))
    lam_pos[:, f], lam_vel[:, f] = a, b
    v0 = pr.vel[:, f].copy()
    h = pr.solver(configs.NU, v0)
    try:
        h.adjoint_record(steps, every)
        end = h.state()
        _, gv, gnu = h.adjoint_backward(lam_pos, lam_vel)
        _, gv2, gnu2 = h.adjoint_backward(lam_pos, lam_vel)
        again = h.state()
    finally:
        h.close()
    assert all(np.array_equal(end[k], again[k]) for k in ("typ", "pos", "vel", "prs"))
    # the same up to the order of the double atomic adds
    assert np.max(np.abs(gv - gv2)) <= 1e-8 * np.max(np.abs(gv)) and abs(gnu - gnu2) <= 1e-8 * abs(gnu)

    def value(nu, v):
        st = pr.run(nu, v)
        return _dot(a, st["pos"][:, f]) + _dot(b, st["vel"][:, f])

    eps = 1e-6 * float(np.sqrt(np.mean(v0 ** 2)))
    fd = (value(configs.NU, v0 + eps * d) - value(configs.NU, v0 - eps * d)) / (2 * eps)
    assert abs(fd - _dot(gv[:, f], d)) <= 1e-3 * abs(fd), (fd, _dot(gv[:, f], d))
    hn = 1e-4 * configs.NU
    fd = (value(configs.NU + hn, v0) - value(configs.NU - hn, v0)) / (2 * hn)
    assert abs(fd - gnu) <= 1e-3 * abs(fd), (fd, gnu)


@pytest.mark.parametrize("block,tank,every", [
    ((8, 6, 10), (20, 10, 20), 6),      # one segment
    ((8, 6, 10), (20, 10, 20), 4),      # the last one short
    ((23, 17, 13), (40, 17, 15), 3),
])
def test_recording_leaves_the_handle_as_the_same_steps_do(block, tank, every):
    """The last segment runs with the recording kernels: state, mirrors and counters, the steps
    that follow, and the gradient are those of ordinary steps and a replay (diagnostics on)."""
    l0, n = 0.02, 6
    pr = RolloutProblem(SceneDesc(l0, tuple(t * l0 for t in tank), block, seed=6, vel_sigma=0.2,
                                  vel_seed=3), dt=2e-4, steps=n, every=every)
    v0 = pr.vel[:, pr.fluid].copy()
    hs = [pr.solver(configs.NU, v0) for _ in range(3)]
    lam = np.zeros((3, pr.typ.shape[0]))
    lam[:, pr.fluid] = np.random.default_rng(8).standard_normal((3, pr.fluid.size))

    def same(a, b):
        x, y = a.state(), b.state()
        for k in ("typ", "pos", "vel", "acc", "prs", "pav"):
            assert np.array_equal(x[k], y[k]), k
        for k in ("steps", "n_fluid_alive", "n_mirror_1", "n_mirror_2"):
            assert a.counters()[k] == b.counters()[k], k
        for w in (2, 1, 0):
            p, q = a.mirrors(w), b.mirrors(w)
            assert all(np.array_equal(p[k], q[k]) for k in ("slot", "pos")), w

    try:
        stepped, taped, replayed = hs
        replayed.set_option(L.OPT_DIAG, 1)
        for h in hs:
            h.step(2)   # a pending step end before the recording
        stepped.step(n)
        grads = []
        for h in (taped, replayed):
            h.adjoint_record(n, every)
            grads.append(h.adjoint_backward(lam, lam) if h is replayed else None)
        same(stepped, taped)
        grads[0] = taped.adjoint_backward(lam, lam)
        for a, b in zip(*grads):
            assert np.max(np.abs(np.subtract(a, b))) <= 1e-8 * np.max(np.abs(a))
        for h in hs:
            h.step(3)
        same(stepped, taped)
        same(stepped, replayed)
        # a handle that has moved on since replays the whole rollout, as ever
        grads = [h.adjoint_backward(lam, lam) for h in (taped, replayed)]
        for a, b in zip(*grads):
            assert np.max(np.abs(np.subtract(a, b))) <= 1e-8 * np.max(np.abs(a))
        same(taped, replayed)
    finally:
        for h in hs:
            h.close()
