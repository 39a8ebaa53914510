"""Walls whose normal is NaN: equal to no normal, each registers once and leaves the other walls'
mirrors alone, whether the walls are told apart by class or, once they have moved, by normal.
"""
from __future__ import annotations

import numpy as np
import pytest

from mps_cuda_b200 import F32, MPS, SceneDesc, dambreak, dambreak_params
from mps_cuda_b200 import _lib as L
from oracle.oracle import Oracle, params_from

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nans", [1, 4, 15])  # one, several, more than a particle registers
@pytest.mark.parametrize("block", [
    (9, 8, 11),    # a warp per particle
    (23, 17, 13),  # 16 lanes
    (23, 23, 24),  # eight lanes
])
@pytest.mark.parametrize("moving", [False, True])
def test_walls_with_nan_normals(block, nans, moving):
    l0 = 0.02
    tank = tuple(b + 4 for b in block)
    d = SceneDesc(l0, tuple(t * l0 for t in tank), block, seed=5, vel_sigma=0.3)
    sc = dambreak(d)
    yy, zz = np.meshgrid((np.arange(tank[1]) + 0.5) * l0, (np.arange(block[2]) + 0.5) * l0)
    plate = np.stack([np.full(yy.size, (block[0] + 0.7) * l0), yy.ravel(), zz.ravel()])
    side = np.tile([[-1.0], [0.0], [0.0]], (1, yy.size))
    # the walls nearest to the plate's point (y, z) = (4.5, 4.5) spacings
    near = np.argsort(np.hypot(yy.ravel() - 4.5 * l0, zz.ravel() - 4.5 * l0), kind="stable")[:nans]
    side[:, near] = np.nan
    typ = np.concatenate([sc["typ"], np.full(yy.size, L.OBJ, np.int8)])
    args = [typ, *(np.concatenate(v, 1).astype(np.float32) for v in (
        (sc["pos"], plate), (sc["vel"], np.zeros_like(plate)), (sc["nrm"], side)))]
    p = dambreak_params(d, dt=2e-4, precision=F32)
    g, o = MPS(p, *args), Oracle(params_from(p), *args)
    try:
        if moving:
            for h in (g, o):
                h.set_wall_motion(L.OBJ, ((block[0] + 0.7) * l0, 0.1, 0.1), (0.0, 0.0, 1.0), 0.0,
                                  (-0.02, 0.0, 0.0))
        g.step(2)
        o.step(2)
        a, b = g.state(), o.state()
        for k in ("typ", "pos", "vel", "prs", "pav"):
            assert np.array_equal(a[k], b[k]), k
        # a mirror through a NaN plane lies nowhere: the cull removes it or it acts on nothing
        real = []
        for m in (g.mirrors(2), o.mirrors()):
            at = ~np.isnan(m["pos"]).any(0)
            real.append((m["slot"][at], m["pos"][:, at]))
        assert np.array_equal(real[0][0], real[1][0]) and np.array_equal(real[0][1], real[1][1])
    finally:
        g.close()
        o.close()
