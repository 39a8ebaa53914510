"""Batches on both sides of the line from eight lanes per particle to one thread in ChkCol/MkPrs,
PrsGrdTrm and mirror generation, against the CPU oracle; the sequence of methods on both sides of its
line for mirror generation; and what a step of a batch costs across the first line.
"""
from __future__ import annotations

import time

import numpy as np
import pytest

from mps_cuda_b200 import F32, F64, MPS, MPSBatch, SceneDesc, configs, dambreak, dambreak_params
from mps_cuda_b200 import _lib as L
from oracle.oracle import Oracle, params_from

pytestmark = pytest.mark.gpu

L0 = 0.02
FIELDS = ("typ", "pos", "vel", "prs", "pav")


def _scene(block, prec, seed=5, dt=2e-4):
    d = SceneDesc(L0, tuple((b + 3) * L0 for b in block), block, seed=seed, vel_sigma=0.3)
    sc = dambreak(d)
    real = np.float64 if prec == F64 else np.float32
    return (dambreak_params(d, dt=dt, precision=prec),
            [sc["typ"], *(sc[k].astype(real) for k in ("pos", "vel", "nrm"))])


def _batch(scenes):
    join = [np.concatenate([a[k] for _, a in scenes], axis=-1) for k in range(4)]
    return MPSBatch([p for p, _ in scenes], *join, counts=[a[0].size for _, a in scenes])


@pytest.mark.parametrize("prec", [F32, F64])
@pytest.mark.parametrize("blocks", [
    [(32, 32, 40), (31, 33, 40), (1, 1, 40)],             # 81920 in all: eight lanes
    [(32, 32, 40), (1, 1, 1), (32, 32, 40), (7, 9, 11)],  # 82614: one thread
])
def test_a_batch_equals_the_oracles(blocks, prec):
    scenes = [_scene(b, prec, seed=3 + i) for i, b in enumerate(blocks)]
    h = _batch(scenes)
    try:
        h.step(2)
        st, at = h.state(), 0
        for p, args in scenes:
            o = Oracle(params_from(p), *args)
            o.step(2)
            one, n = o.state(), args[0].size
            for k in FIELDS:
                assert np.array_equal(st[k][..., at:at + n], one[k]), k
            o.close()
            at += n
    finally:
        h.close()


@pytest.mark.parametrize("prec", [F32, F64])
@pytest.mark.parametrize("block", [
    (40, 44, 64),  # 112640: the last size of eight lanes where mirror generation runs by itself
    (43, 47, 56),  # 113176
])
def test_the_methods_equal_the_oracle(block, prec):
    p, args = _scene(block, prec)
    g, o = MPS(p, *args), Oracle(params_from(p), *args)
    try:
        g.step_by_methods()
        o.step(1)
        a, b = g.state(), o.state()
        for k in FIELDS:
            assert np.array_equal(a[k], b[k]), k
    finally:
        g.close()
        o.close()


def test_a_batch_beyond_the_line_steps_with_one_thread_throughout():
    """62 133 particles in eight scenes step in 531 us, 101 575 in twelve in 600 with one thread per
    particle throughout and in 687 with eight lanes in mirror generation alone: 1.13 and 1.29 times."""
    handles = []
    try:
        for n in (8, 12):
            scenes = configs.batched_scenes(n, seed=11)
            parts = []
            for d, dt in scenes:
                sc = dambreak(d)
                parts.append((dambreak_params(d, dt=dt, precision=F32),
                              [sc["typ"], *(sc[k].astype(np.float32) for k in ("pos", "vel", "nrm"))]))
            h = _batch(parts)
            h.set_option(L.OPT_GRAPH, 1)
            handles.append(h)
        states, best = [h.state() for h in handles], [float("inf")] * 2
        for _ in range(8):
            for i, h in enumerate(handles):
                h.set_state(**states[i])
                h.step(3)
                h.synchronize()
                t0 = time.perf_counter()
                h.step(20)
                h.synchronize()
                best[i] = min(best[i], time.perf_counter() - t0)
        assert best[1] < 1.21 * best[0], best
    finally:
        for h in handles:
            h.close()
