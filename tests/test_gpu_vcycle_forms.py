"""The launch forms of one V-cycle give the same bits on grids where a form's
index rules can go wrong: rows of one cell, odd and even rows, single planes,
two-cell grids, levels around the sizes at which a form takes over.

Default: the pair tail (levels of at most 1024 cells in one block), residual
and restriction in one launch below PFGPU_FUSE_CELLS, the zero-guess red sweep
done by whoever writes the right-hand side.  Compared with the generic tail in
global memory (PFGPU_TAIL_SMEM=0), every level on the grid kernels
(PFGPU_TAIL_CELLS=1), residual and restriction apart (PFGPU_FUSE_CELLS=0) and
the natural layout of the iterates (PFGPU_SPLIT=0)."""

import numpy as np
import pytest

from parflow_b200 import configs
from parflow_b200.problem import SolverSettings

pytestmark = pytest.mark.gpu

ENV = ("PFGPU_TAIL_SMEM", "PFGPU_TAIL_CELLS", "PFGPU_FUSE_CELLS", "PFGPU_SPLIT")
SHAPES = [(1, 1, 2), (2, 1, 1), (1, 37, 5), (2, 2, 2), (3, 5, 7), (16, 16, 4), (17, 15, 4),
          (33, 31, 1), (1, 64, 33), (128, 3, 11), (65, 63, 9), (1, 45, 45)]


@pytest.fixture(scope="module")
def solver():
    import torch

    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from parflow_b200 import solver as s

    return s


def _pc(solver, prob, precision, monkeypatch, env):
    for k in ENV:
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    s = solver.RichardsGPU(prob, precision=precision)
    rng = np.random.default_rng(11)
    p = prob.initial_pressure() + 0.1 * rng.standard_normal(prob.shape)
    s.pc_setup(p, prob.dt)
    z = s.pc_apply(rng.standard_normal(prob.shape))
    z2 = s.pc_apply(z)
    s.close()
    return np.concatenate([z.ravel(), z2.ravel()])


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed16"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_forms_bitwise_equal(solver, monkeypatch, shape, precision, symmetric):
    nx, ny, nz = shape
    prob = configs.box(nx=nx, ny=ny, nz=nz, nsteps=1,
                       solver=SolverSettings(mg_smoother_symmetric=symmetric))
    ref = _pc(solver, prob, precision, monkeypatch, {})
    assert np.isfinite(ref).all() and np.abs(ref).max() > 0
    for env in ({"PFGPU_TAIL_SMEM": "0"}, {"PFGPU_TAIL_CELLS": "1"}, {"PFGPU_FUSE_CELLS": "0"},
                {"PFGPU_TAIL_CELLS": "1", "PFGPU_FUSE_CELLS": "0"}, {"PFGPU_SPLIT": "0"}):
        z = _pc(solver, prob, precision, monkeypatch, env)
        assert np.array_equal(z, ref), env


@pytest.mark.parametrize("precision", ["fp64", "mixed16"])
def test_tail_moves_with_max_iter(solver, monkeypatch, precision):
    """A grid that is all tail: MGSemi.MaxIter 2 takes level 0 out of it, back
    to 1 leaves it out; the packed operators follow without a new setup."""
    for k in ENV:
        monkeypatch.delenv(k, raising=False)
    prob = configs.box(nx=12, ny=10, nz=8, nsteps=1)
    s = solver.RichardsGPU(prob, precision=precision)
    rng = np.random.default_rng(12)
    p = prob.initial_pressure() + 0.1 * rng.standard_normal(prob.shape)
    r = rng.standard_normal(prob.shape)
    s.pc_setup(p, prob.dt)
    z = s.pc_apply(r)
    assert s.lib.pfgpu_set_mg_max_iter(s.h, 2) == 0
    s.pc_apply(r)
    assert s.lib.pfgpu_set_mg_max_iter(s.h, 1) == 0
    assert np.array_equal(s.pc_apply(r), z)
    s.close()


@pytest.mark.parametrize("shape", [(1, 45, 45), (2, 32, 32)], ids=lambda s: "x".join(map(str, s)))
def test_tail_setup_matches_oracle(solver, monkeypatch, shape):
    """FP64 hierarchies whose first level is all but as large as the one-block
    setup takes: with rows of one cell the ghost columns do not fit the shared
    memory beside the operators, and the generic setup feeds the packed tail."""
    from oracle.oracle import Oracle

    for k in ENV:
        monkeypatch.delenv(k, raising=False)
    nx, ny, nz = shape
    prob = configs.box(nx=nx, ny=ny, nz=nz, nsteps=1)
    rng = np.random.default_rng(13)
    p = prob.initial_pressure() + 0.1 * rng.standard_normal(prob.shape)
    r = rng.standard_normal(prob.shape)
    s = solver.RichardsGPU(prob)
    levels = s.mg_levels()
    cells = sum(a * b * c for a, b, c, _ in levels)
    ghosts = sum(b * c for _, b, c, _ in levels)
    assert levels[0][0] * levels[0][1] * levels[0][2] <= 2048
    assert (8 * (4 * cells + ghosts) > 160 * 1024) == (nx == 1)
    s.pc_setup(p, prob.dt)
    z = s.pc_apply(r)
    s.close()
    orc = Oracle(prob)
    mg = orc.mg()
    mg.setup(orc.jacobian(p, prob.dt, symm=1))
    want = mg.apply(r)
    assert np.abs(z - want).max() <= 1e-12 * np.abs(want).max()


def test_full_jacobian_comes_and_goes(solver, monkeypatch):
    """FullJacobian, back, and again: the second solve is not a captured one that
    holds the first one's arrays; its pressures are a new handle's."""
    for k in ENV:
        monkeypatch.delenv(k, raising=False)
    prob = configs.box(nx=20, ny=14, nz=9, nsteps=1)
    t, dt = prob.time_plan()[0]
    p0 = prob.initial_pressure()

    def step(s):
        s.set_time(t)
        s.set_pressure(p0)
        s.advance(1, dt)
        return s.get_pressure()

    s = solver.RichardsGPU(prob)
    symmetric = step(s)
    got = []
    for _ in range(2):
        assert s.lib.pfgpu_set_pc_matrix(s.h, 1) == 0
        got.append(step(s))
        assert s.lib.pfgpu_set_pc_matrix(s.h, 0) == 0
        # (level 0 stays out of the tail: equal up to the V-cycle's rounding)
        assert np.abs(step(s) - symmetric).max() <= 1e-9 * np.abs(symmetric).max()
    s.close()
    fresh = solver.RichardsGPU(prob)
    assert fresh.lib.pfgpu_set_pc_matrix(fresh.h, 1) == 0
    want = step(fresh)
    fresh.close()
    assert np.array_equal(got[0], want) and np.array_equal(got[1], want)
