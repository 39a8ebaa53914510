"""Scenes whose grid has 4096 buckets or more along an axis.

The walks with several lanes per particle do not cover them; the kernels with one thread per
particle serve them at every size, alone and in a batch.
"""
from __future__ import annotations

import time

import numpy as np
import pytest

from mps_cuda_b200 import F32, F64, MPS, MPSBatch, SceneDesc, dambreak, dambreak_params
from oracle.oracle import Oracle, params_from

pytestmark = pytest.mark.gpu

L0 = 0.02
BLOCKS = [(9, 8, 11), (23, 17, 13), (23, 23, 24)]  # a warp, 16 and eight lanes where they serve
FIELDS = ("typ", "pos", "vel", "prs", "pav")


def _scene(block, buckets, prec):
    """The column at the low end of a domain of that many buckets along x (3.1 spacings each)."""
    d = SceneDesc(L0, tuple((b + 3) * L0 for b in block), block, seed=5, vel_sigma=0.3)
    sc = dambreak(d)
    real = np.float64 if prec == F64 else np.float32
    p = dambreak_params(d, dt=2e-4, precision=prec)
    p.max[0] = p.min[0] + (buckets - 4.5) * 3.1 * L0
    return p, [sc["typ"], *(sc[k].astype(real) for k in ("pos", "vel", "nrm"))]


@pytest.mark.parametrize("prec", [F32, F64])
@pytest.mark.parametrize("block", BLOCKS)
@pytest.mark.parametrize("buckets", [4094, 4096, 4100])
def test_steps_equal_the_oracle(block, prec, buckets):
    p, args = _scene(block, buckets, prec)
    g, o = MPS(p, *args), Oracle(params_from(p), *args)
    try:
        for n in (1, 3):
            g.step(n)
            o.step(n)
            a, b = g.state(), o.state()
            for k in FIELDS:
                assert np.array_equal(a[k], b[k]), (n, k)
    finally:
        g.close()
        o.close()


def test_a_long_scene_in_a_batch_leaves_the_others_as_they_are():
    p1, a1 = _scene(BLOCKS[0], 4100, F32)
    p2, a2 = _scene(BLOCKS[0], 60, F32)
    join = lambda k: np.concatenate([a2[k], a1[k], a2[k]], axis=-1)
    b = MPSBatch([p2, p1, p2], *(join(k) for k in range(4)), counts=[x[0].size for x in (a2, a1, a2)])
    o = [Oracle(params_from(p), *a) for p, a in ((p2, a2), (p1, a1), (p2, a2))]
    try:
        b.step(3)
        st, at = b.state(), 0
        for h in o:
            h.step(3)
            one = h.state()
            n = one["typ"].size
            for k in FIELDS:
                assert np.array_equal(st[k][..., at:at + n], one[k]), k
            at += n
    finally:
        b.close()
        for h in o:
            h.close()


def test_a_long_grid_costs_no_lanes():
    """64 000 particles step about as fast with one thread each as with eight lanes; one working
    lane of a group of eight takes several times as long."""
    handles = []
    try:
        for buckets in (4080, 4110):
            p, args = _scene((40, 40, 40), buckets, F32)
            handles.append(MPS(p, *args))
        best = [float("inf")] * 2
        for _ in range(7):
            for i, h in enumerate(handles):
                h.step(2)
                h.synchronize()
                t0 = time.perf_counter()
                h.step(20)
                h.synchronize()
                best[i] = min(best[i], time.perf_counter() - t0)
        assert best[1] < 1.6 * best[0], best
    finally:
        for h in handles:
            h.close()
