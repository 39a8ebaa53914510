"""Autotuning where several lanes per particle leave a kernel one shape: nothing is picked for it, and
nothing that was picked reaches handles that run other kernels.
"""
from __future__ import annotations

import numpy as np
import pytest

from mps_cuda_b200 import F32, F64, MPS, SceneDesc, dambreak, dambreak_params
from mps_cuda_b200 import _lib as L

pytestmark = pytest.mark.gpu

L0 = 0.02
SETTINGS = (L.OPT_BLOCK, L.OPT_CANDIDATE_BATCH, L.OPT_REGISTER_BOUND, L.OPT_STAGING)


def _handle(block, prec):
    d = SceneDesc(L0, tuple((b + 3) * L0 for b in block), block, seed=5, vel_sigma=0.3)
    sc = dambreak(d)
    real = np.float64 if prec == F64 else np.float32
    return MPS(dambreak_params(d, dt=2e-4, precision=prec), sc["typ"],
               *(sc[k].astype(real) for k in ("pos", "vel", "nrm")))


@pytest.mark.parametrize("prec,block,other", [
    (F32, (9, 8, 11), (9, 9, 11)),        # a warp each
    (F32, (23, 17, 13), None),            # 16 lanes
    (F64, (23, 23, 24), (13, 29, 23)),    # 12 696: eight lanes; 8 671: 16
    (F64, (35, 35, 34), (43, 31, 43)),    # 41 650: eight lanes in pass A as well; 57 319: not
    (F32, (40, 42, 42), (46, 46, 47)),    # 70 560: eight lanes in ChkCol/MkPrs; 99 452: nowhere
])
def test_nothing_is_picked_for_a_kernel_of_one_shape(prec, block, other):
    g = _handle(block, prec)
    before = g.state()
    chosen = g.autotune(1)
    assert [chosen[k] for k in ("pass_b", "pass_c", "gen_cull")] == [128] * 3
    assert chosen["register_bound"] & 3 == 0
    if block != (40, 42, 42):
        assert chosen["pass_a"] == 128 and chosen["candidate_batch"] == 4
        assert chosen["register_bound"] == 0
    after = g.state()
    assert all(np.array_equal(after[k], before[k]) for k in before)
    picked = [g.get_option(k) for k in SETTINGS]
    g.close()
    if other:
        h = _handle(other, prec)
        same = block == (9, 8, 11)  # the same kernels, or other ones with settings of their own
        assert [h.get_option(k) for k in SETTINGS] == (picked if same else [128, 4, 0, L.STAGE_GLOBAL])
        h.close()
