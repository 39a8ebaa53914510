"""The neighbour passes with several lanes per particle (mps_group.cuh) against the CPU oracle.

Small scenes run the passes with a warp, 16 or eight lanes per particle, larger ones with one thread
(Solver::group_lanes); every path must give the oracle's state bit for bit. The blocks have odd
sides, so that a warp's particles span bucket rows and the last warp is ragged; the sizes lie on
both sides of the lines between a warp, 16 and eight lanes, and on the line of one thread.
"""
from __future__ import annotations

import numpy as np
import pytest

from mps_cuda_b200 import F32, F32_N64, F64, MPS, SceneDesc, dambreak, dambreak_params
from mps_cuda_b200 import _lib as L
from oracle.oracle import Oracle, params_from

pytestmark = pytest.mark.gpu

FIELDS = ("typ", "pos", "vel", "prs", "pav")


def _pair(block, tank, prec, l0=0.02, dt=2e-4, **desc):
    d = SceneDesc(l0, tuple(t * l0 for t in tank), block, seed=5, vel_sigma=0.3, **desc)
    sc = dambreak(d)
    p = dambreak_params(d, dt=dt, precision=prec)
    real = np.float64 if prec == F64 else np.float32
    args = [sc["typ"], *(sc[k].astype(real) for k in ("pos", "vel", "nrm"))]
    return MPS(p, *args), Oracle(params_from(p), *args)


def _steps(g, o, n, where):
    g.step(n)
    o.step(n)
    a, b = g.state(), o.state()
    for k in FIELDS:
        assert np.array_equal(a[k], b[k]), (where, k)


@pytest.mark.parametrize("prec", [F32, F64, F32_N64])
@pytest.mark.parametrize("block,tank", [
    ((1, 1, 2), (5, 4, 6)),       # two particles, a nearly empty warp
    ((3, 7, 11), (9, 7, 13)),     # 231
    ((10, 15, 20), (14, 16, 22)),  # 3000: the last size of a warp each in FP64
    ((17, 13, 19), (30, 14, 21)),  # 4199: a warp each in FP32, 16 lanes in FP64
    ((20, 11, 20), (24, 12, 23)),  # 4400: the last size of a warp each in FP32
    ((25, 8, 25), (31, 9, 27)),   # 5000: the last size of the one-launch bucket builds
    ((23, 17, 13), (40, 17, 15)),  # 5083: 16 lanes each
    ((16, 24, 32), (20, 24, 34)),  # 12288: the last size of 16 lanes each
    ((23, 23, 24), (28, 24, 26)),  # 12696: eight lanes each
])
def test_odd_scenes_equal_the_oracle(block, tank, prec):
    g, o = _pair(block, tank, prec)
    try:
        _steps(g, o, 1, "first")
        _steps(g, o, 6, "later")
        a, b = g.mirrors(2), o.mirrors()
        assert np.array_equal(a["slot"], b["slot"]) and np.array_equal(a["pos"], b["pos"])
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("opts", [
    {L.OPT_DIAG: 1}, {L.OPT_LIST_CAPACITY: 9}, {L.OPT_GRADIENT: L.GRAD_CORRECTED}, {L.OPT_CELL_SKIP: 0},
])
@pytest.mark.parametrize("block", [(9, 8, 11), (23, 17, 13), (23, 23, 24)])
def test_options_equal_the_oracle(block, opts):
    tank = tuple(b + 3 for b in block)
    g, o = _pair(block, tank, F32)
    try:
        for k, v in opts.items():
            g.set_option(k, v)
        if L.OPT_GRADIENT in opts:
            o.set_gradient(1)
        _steps(g, o, 3, opts)
        if L.OPT_DIAG in opts:
            a, b, fl = g.diag(), o.diag(), o.state()["typ"] == L.FLD
            for k in L.DIAG_COLUMNS:
                assert np.array_equal(a[k][fl], b[k][fl]), k
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("block", [(9, 8, 11), (23, 17, 13), (23, 23, 24)])
def test_scales_outside_the_fast_arithmetic_equal_the_oracle(block):
    """A spacing below 2^-20 takes the walk of one lane per particle inside the same kernels."""
    tank = tuple(b + 3 for b in block)
    g, o = _pair(block, tank, F32, l0=2e-7, dt=1e-10)
    try:
        _steps(g, o, 3, block)
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("shift", [0.0, 1e-6])
def test_nearly_coincident_particles_equal_the_oracle(shift):
    """Pairs closer than l0 / 1024 leave the fast arithmetic; coincident ones give infinities."""
    g, o = _pair((9, 8, 11), (14, 8, 14), F32)
    try:
        st = o.state()
        pos = st["pos"].copy()
        for i, j in ((100, 101), (400, 470)):
            pos[:, j] = pos[:, i] + np.float32(shift)
        g.set_state(pos=pos)
        o.set_state(pos=pos)
        g.step(1)
        o.step(1)
        a, b = g.state(), o.state()
        for k in FIELDS:
            assert np.array_equal(a[k], b[k], equal_nan=k != "typ"), k
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("block", [(9, 8, 11), (23, 17, 13), (23, 23, 24)])
def test_walls_that_moved_and_stopped_equal_the_oracle(block):
    """Walls at rest are told apart by class; a wall that has moved is not, nor once it stops."""
    l0 = 0.02
    tank = tuple(b + 4 for b in block)
    d = SceneDesc(l0, tuple(t * l0 for t in tank), block, seed=5, vel_sigma=0.3)
    sc = dambreak(d)
    yy, zz = np.meshgrid((np.arange(tank[1]) + 0.5) * l0, (np.arange(block[2]) + 0.5) * l0)
    plate = np.stack([np.full(yy.size, (block[0] + 0.7) * l0), yy.ravel(), zz.ravel()])
    side = np.tile([[-1.0], [0.0], [0.0]], (1, yy.size))
    typ = np.concatenate([sc["typ"], np.full(yy.size, L.OBJ, np.int8)])
    args = [typ, *(np.concatenate(v, 1).astype(np.float32) for v in (
        (sc["pos"], plate), (sc["vel"], np.zeros_like(plate)), (sc["nrm"], side)))]
    p = dambreak_params(d, dt=2e-4, precision=F32)
    g, o = MPS(p, *args), Oracle(params_from(p), *args)
    try:
        _steps(g, o, 2, "before")
        for omega, vx in ((3.0, -0.5), (0.0, 0.0)):
            for h in (g, o):
                h.set_wall_motion(L.OBJ, ((block[0] + 0.7) * l0, 0.1, 0.1), (0.0, 0.0, 1.0), omega,
                                  (vx, 0.0, 0.0))
            _steps(g, o, 4, (omega, vx))
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("prec", [F32, F64])
@pytest.mark.parametrize("block", [(9, 8, 11), (23, 17, 13), (23, 23, 24)])
def test_many_wall_normals_equal_the_oracle(block, prec):
    """A rough plate: 14 normals within reach of a particle, more than a particle registers."""
    l0 = 0.02
    tank = tuple(b + 4 for b in block)
    d = SceneDesc(l0, tuple(t * l0 for t in tank), block, seed=5, vel_sigma=0.3)
    sc = dambreak(d)
    yy, zz = np.meshgrid((np.arange(tank[1]) + 0.5) * l0, (np.arange(block[2]) + 0.5) * l0)
    plate = np.stack([np.full(yy.size, (block[0] + 0.7) * l0), yy.ravel(), zz.ravel()])
    tilt = np.random.default_rng(2).uniform(-0.2, 0.2, (14, 2))
    side = np.stack([-np.ones(14), tilt[:, 0], tilt[:, 1]])
    side = (side / np.linalg.norm(side, axis=0))[:, np.arange(yy.size) % 14]
    real = np.float64 if prec == F64 else np.float32
    typ = np.concatenate([sc["typ"], np.full(yy.size, L.OBJ, np.int8)])
    args = [typ, *(np.concatenate(v, 1).astype(real) for v in (
        (sc["pos"], plate), (sc["vel"], np.zeros_like(plate)), (sc["nrm"], side)))]
    p = dambreak_params(d, dt=2e-4, precision=prec)
    g, o = MPS(p, *args), Oracle(params_from(p), *args)
    try:
        _steps(g, o, 3, block)
        a, b = g.mirrors(2), o.mirrors()
        assert np.array_equal(a["slot"], b["slot"]) and np.array_equal(a["pos"], b["pos"])
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("corrected", [0, 1])
@pytest.mark.parametrize("prec", [F32, F64, F32_N64])
@pytest.mark.parametrize("block", [(9, 8, 11), (23, 17, 13), (23, 23, 24)])
def test_methods_one_by_one_equal_the_oracle(block, prec, corrected):
    """Every method on its own, in the reference's order and then without the bucket builds that
    follow a move: the lists are then older than the positions, and one thread walks them."""
    tank = tuple(b + 3 for b in block)
    g, o = _pair(block, tank, prec)
    step = [0, 2, 3, 4, 5, 6, 0, 7, 0, 8, 2, 3, 4, 9, 10]
    stale = [2, 3, 4, 5, 6, 7, 8, 2, 3, 4, 9, 10]
    try:
        if corrected:
            g.set_option(L.OPT_GRADIENT, L.GRAD_CORRECTED)
            o.set_gradient(1)
        for phases in (step, step, [0] + stale):
            for ph in phases:
                g.phase(ph)
                o.phase(ph)
                a, b = g.state(), o.state()
                for k in FIELDS + ("acc",):
                    assert np.array_equal(a[k], b[k], equal_nan=k != "typ"), (ph, k)
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("prec", [F32, F64])
@pytest.mark.parametrize("block", [
    (40, 35, 40),   # 56000 and 65536: the last sizes of several lanes in pass A, FP64 and FP32
    (32, 32, 64),
    (40, 32, 64),   # 81920: the last size of several lanes in passes B and C
    (43, 41, 47),   # 82861: their lists have the one-thread layout
])
def test_the_lines_of_one_thread_equal_the_oracle(block, prec):
    g, o = _pair(block, tuple(b + 3 for b in block), prec)
    try:
        _steps(g, o, 2, block)
    finally:
        g.close()
        o.close()
