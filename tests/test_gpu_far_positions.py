"""Particles that a state places beyond the grid, by as little as a bucket and as far as infinity.

Each gets the nearest bucket (the number of buckets to it need not fit an int), neighbours keep
their walks, and the step deletes it, as the oracle does. Bucket rows of even and odd length, every
number of lanes per particle, one-launch bucket builds and the others.
"""
from __future__ import annotations

import numpy as np
import pytest

from mps_cuda_b200 import F32, F64, MPS, SceneDesc, dambreak, dambreak_params
from mps_cuda_b200 import _lib as L
from oracle.oracle import Oracle, params_from

pytestmark = pytest.mark.gpu

L0 = 0.02
FIELDS = ("typ", "pos", "vel", "prs", "pav")
BLOCKS = [
    (9, 8, 11),    # 8 buckets along x; a warp per particle
    (11, 8, 9),    # 9 buckets along x
    (23, 17, 13),  # 16 lanes
    (23, 23, 24),  # eight lanes
    (43, 41, 47),  # one thread
]


def _pair(block, prec):
    d = SceneDesc(L0, tuple((b + 3) * L0 for b in block), block, seed=5, vel_sigma=0.3)
    sc = dambreak(d)
    real = np.float64 if prec == F64 else np.float32
    args = [sc["typ"], *(sc[k].astype(real) for k in ("pos", "vel", "nrm"))]
    p = dambreak_params(d, dt=2e-4, precision=prec)
    return MPS(p, *args), Oracle(params_from(p), *args), args[1]


def _misplaced(pos):
    bad = pos.copy()
    big = 1e30 if pos.dtype == np.float32 else 1e300
    for axis in range(3):
        for k, v in enumerate((0.4, 40.0, 1.3e8, big, np.inf)):
            bad[axis, 31 * (5 * axis + k) + 2] = -v - 6.5 * L0
            bad[axis, 31 * (5 * axis + k) + 17] = v + (pos[axis].max() + 7.0 * L0)
    return bad


@pytest.mark.parametrize("prec", [F32, F64])
@pytest.mark.parametrize("block", BLOCKS)
def test_steps_equal_the_oracle(block, prec):
    g, o, pos = _pair(block, prec)
    try:
        bad = _misplaced(pos)
        g.set_state(pos=bad)
        o.set_state(pos=bad)
        for n in (1, 2):
            g.step(n)
            o.step(n)
            a, b = g.state(), o.state()
            for k in FIELDS:
                assert np.array_equal(a[k], b[k], equal_nan=k != "typ"), (n, k)
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("staging", [L.STAGE_GLOBAL, L.STAGE_POSITIONS])
@pytest.mark.parametrize("block", BLOCKS)
def test_other_routes_to_a_step_equal_the_plain_one(block, staging):
    """Graphs, diagnostics, a staged pass A, and the methods one by one."""
    hs = []
    try:
        for opt in ({}, {L.OPT_GRAPH: 1}, {L.OPT_DIAG: 1}, {L.OPT_CELL_SKIP: 0}, None):
            g, o, pos = _pair(block, F32)
            o.close()
            hs.append(g)
            g.set_option(L.OPT_STAGING, staging)
            for k, v in (opt or {}).items():
                g.set_option(k, v)
            g.set_state(pos=_misplaced(pos))
            if opt is None:
                g.step_by_methods()
                g.step_by_methods()
            else:
                g.step(2)
        want = hs[0].state()
        for i, h in enumerate(hs[1:]):
            got = h.state()
            for k in FIELDS:
                assert np.array_equal(got[k], want[k], equal_nan=k != "typ"), (i, k)
    finally:
        for h in hs:
            h.close()
