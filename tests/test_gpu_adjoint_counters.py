"""The error counters of a handle after a recorded rollout: those of the same steps taken plainly."""
from __future__ import annotations

import numpy as np
import pytest

from mps_cuda_b200 import F64, MPS, SceneDesc, dambreak, dambreak_params
from mps_cuda_b200 import _lib as L

pytestmark = pytest.mark.gpu

L0 = 0.02
ERRORS = ("err_mirror_slot", "err_mirror_capacity", "err_cell_range", "err_nan")


def _handle(block):
    """Walls that all face different ways: more planes than a particle has places for, and mirrors
    beyond the grid; and two particles off the grid."""
    d = SceneDesc(L0, tuple((b + 3) * L0 for b in block), block, seed=5, vel_sigma=0.3)
    sc = dambreak(d)
    nrm = np.random.default_rng(3).normal(size=sc["nrm"].shape) * (sc["typ"] != L.FLD)
    nrm = nrm / np.maximum(np.linalg.norm(nrm, axis=0), 1e-30)
    h = MPS(dambreak_params(d, dt=2e-4, precision=F64), sc["typ"], sc["pos"], sc["vel"], nrm)
    pos = h.state()["pos"]
    pos[0, 100:102] = (-1.0, 5.0)
    h.set_state(pos=pos)
    return h


def _errors(h):
    c = h.counters()
    return {k: c[k] for k in ERRORS}


@pytest.mark.parametrize("block", [(9, 8, 11), (23, 17, 13)])  # a warp and 16 lanes per particle
@pytest.mark.parametrize("before,looked", [(0, False), (2, False), (2, True)])
@pytest.mark.parametrize("steps,every", [(4, 4), (5, 3), (3, 1)])
def test_recording_counts_each_error_once(steps, every, before, looked, block):
    plain, recorded = _handle(block), _handle(block)
    try:
        for h in (plain, recorded):
            h.step(before)
            if looked:
                h.mirrors(1)  # ends the step: the next mirrors are made already
        plain.step(steps)
        recorded.adjoint_record(steps, every)
        a, b = _errors(plain), _errors(recorded)
        assert a["err_mirror_slot"] > 0 and a["err_cell_range"] > 0
        assert a == b
        plain.step(2)
        recorded.step(2)
        assert _errors(plain) == _errors(recorded)
        a, b = plain.state(), recorded.state()
        for k in a:
            assert np.array_equal(a[k], b[k], equal_nan=k != "typ"), k
    finally:
        plain.close()
        recorded.close()
