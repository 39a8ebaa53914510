"""A rollout recorded again on the same handle after the neighbour lists' capacity has changed.

The second recording's tape has lists of the new capacity: the state it ends in, and its gradient,
are those of a fresh handle at that capacity.
"""
from __future__ import annotations

import numpy as np
import pytest

from mps_cuda_b200 import SceneDesc, configs
from mps_cuda_b200 import _lib as L
from mps_cuda_b200.adjoint import RolloutProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first,second", [(8, 0), (0, 64), (64, 160)])
@pytest.mark.parametrize("block,tank,every", [
    ((8, 6, 10), (20, 10, 20), 4),     # a warp per particle
    ((8, 6, 10), (20, 10, 20), 3),     # two segments
    ((23, 17, 13), (40, 17, 15), 4),   # 16 lanes per particle
])
def test_recording_again_after_a_capacity_change(block, tank, every, first, second):
    l0, n = 0.02, 4
    pr = RolloutProblem(SceneDesc(l0, tuple(t * l0 for t in tank), block, seed=6, vel_sigma=0.2,
                                  vel_seed=3), dt=2e-4, steps=n, every=every)
    v0 = pr.vel[:, pr.fluid].copy()
    lam = np.zeros((3, pr.typ.shape[0]))
    lam[:, pr.fluid] = np.random.default_rng(8).standard_normal((3, pr.fluid.size))
    again, fresh = (pr.solver(configs.NU, v0) for _ in range(2))
    try:
        start = again.state()
        again.set_option(L.OPT_LIST_CAPACITY, first)
        again.adjoint_record(n, every)
        again.set_state(**start)
        for h in (again, fresh):
            h.set_option(L.OPT_LIST_CAPACITY, second)
            h.adjoint_record(n, every)
        a, b = again.state(), fresh.state()
        for k in ("typ", "pos", "vel", "acc", "prs", "pav"):
            assert np.array_equal(a[k], b[k]), k
        # lists of up to 122 lattice neighbours fit 160 entries (0: the most there are), not 64
        if second == 64:
            for h in (again, fresh):
                with pytest.raises(RuntimeError, match="exceeded"):
                    h.adjoint_backward(lam, lam)
        else:
            for p, q in zip(again.adjoint_backward(lam, lam), fresh.adjoint_backward(lam, lam)):
                assert np.max(np.abs(np.subtract(p, q))) <= 1e-8 * np.max(np.abs(q))
    finally:
        again.close()
        fresh.close()
