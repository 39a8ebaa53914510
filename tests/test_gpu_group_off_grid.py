"""Particles off the grid, or at no place at all, among particles that walk in groups of lanes.

One lane walks for such a particle; its neighbours keep their groups, and a handle whose state is
replaced by a good one runs as a handle that never met it.
"""
from __future__ import annotations

import time

import numpy as np
import pytest

from mps_cuda_b200 import F32, F64, MPS, SceneDesc, dambreak, dambreak_params
from oracle.oracle import Oracle, params_from

pytestmark = pytest.mark.gpu

BLOCKS = [(9, 8, 11), (23, 17, 13), (23, 23, 24)]  # a warp, 16 and eight lanes per particle
FIELDS = ("typ", "pos", "vel", "prs", "pav")


def _args(block, prec, l0=0.02):
    d = SceneDesc(l0, tuple((b + 3) * l0 for b in block), block, seed=5, vel_sigma=0.3)
    sc = dambreak(d)
    real = np.float64 if prec == F64 else np.float32
    return (dambreak_params(d, dt=2e-4, precision=prec), sc["typ"],
            *(sc[k].astype(real) for k in ("pos", "vel", "nrm")))


@pytest.mark.parametrize("prec", [F32, F64])
@pytest.mark.parametrize("block", BLOCKS)
def test_particles_at_no_place_equal_the_oracle(block, prec):
    """NaN positions lie in no order with the others: every warp that holds one, and its neighbours,
    must walk as if it were not there."""
    p, *args = _args(block, prec)
    g, o = MPS(p, *args), Oracle(params_from(p), *args)
    try:
        bad = args[1].copy()
        for k, i in enumerate((3, 101, 102, 333, 404, 510)):
            bad[k % 3, i] = np.nan if k % 2 else -np.nan
        bad[:, 600] = np.nan
        g.set_state(pos=bad)
        o.set_state(pos=bad)
        for _ in range(3):
            g.step(1)
            o.step(1)
            a, b = g.state(), o.state()
            for k in FIELDS:
                assert np.array_equal(a[k], b[k], equal_nan=k != "typ"), k
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("value", [np.nan, 1e3])
def test_a_repaired_state_runs_at_full_speed(value):
    p, *args = _args(BLOCKS[2], F32)
    fresh, repaired = MPS(p, *args), MPS(p, *args)
    try:
        bad = args[1].copy()
        bad[0, 100] = value
        good = fresh.state()
        repaired.set_state(pos=bad)
        repaired.step(1)
        repaired.set_state(**good)

        def best(h):
            ts = []
            for _ in range(7):
                h.set_state(**good)
                h.step(1)
                h.synchronize()
                t0 = time.perf_counter()
                h.step(20)
                h.synchronize()
                ts.append(time.perf_counter() - t0)
            return min(ts)

        t_fresh, t_repaired = best(fresh), best(repaired)
        a, b = fresh.state(), repaired.state()
        for k in FIELDS:
            assert np.array_equal(a[k], b[k]), k
        # one lane for each particle takes several times as long
        assert t_repaired < 1.5 * t_fresh, (t_repaired, t_fresh)
    finally:
        fresh.close()
        repaired.close()
