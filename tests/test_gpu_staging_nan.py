"""A staged pass A with NaN positions among the particles of a block.

The staged rows come from the box around the block's particles, which a NaN does not bound; such a
block walks global memory. The particles here share the NaN's bucket row: a NaN gets the first
interior bucket, where misplaced particles of the state lie too.
"""
from __future__ import annotations

import numpy as np
import pytest

from mps_cuda_b200 import F32, F64, MPS, SceneDesc, dambreak, dambreak_params
from mps_cuda_b200 import _lib as L
from oracle.oracle import Oracle, params_from

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [F32, F64])
@pytest.mark.parametrize("mode", [L.STAGE_POSITIONS, L.STAGE_VELOCITIES])
def test_nan_in_a_staged_block(mode, prec):
    l0, block = 0.02, (9, 8, 11)
    d = SceneDesc(l0, tuple((b + 3) * l0 for b in block), block, seed=5, vel_sigma=0.3)
    sc = dambreak(d)
    real = np.float64 if prec == F64 else np.float32
    args = [sc["typ"], *(sc[k].astype(real) for k in ("pos", "vel", "nrm"))]
    p = dambreak_params(d, dt=2e-4, precision=prec)
    g, o = MPS(p, *args), Oracle(params_from(p), *args)
    try:
        bad = args[1].copy()
        rng = np.random.default_rng(4)
        # sixty particles in the lowest bucket row, 3.1 spacings high and deep, and up to three
        # buckets along x; NaN ones among them
        bad[1:, :60] = -rng.uniform(0.1, 3.0, (2, 60)) * l0
        bad[0, :60] = rng.uniform(-3.0, 6.0, 60) * l0
        for k, i in enumerate((5, 6, 20, 41)):
            bad[k % 3, i] = np.nan
        for h in (g, o):
            h.set_state(pos=bad)
        g.set_option(L.OPT_STAGING, mode)
        for _ in range(2):
            g.step(1)
            o.step(1)
            a, b = g.state(), o.state()
            for k in ("typ", "pos", "vel", "prs", "pav"):
                assert np.array_equal(a[k], b[k], equal_nan=k != "typ"), k
    finally:
        g.close()
        o.close()
