"""A timestep of two million cells and one (odd) on the forms that only grids of
this size take: march residual and Jacobian, with the trial step formed in the
van Genuchten pass, residual and restriction in two launches on the finest
levels.  Each runs in a child process with one form switched off; the
pressures are the same bits, and the residual that ended the solve is that of
the pressure it returned."""

import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import json, sys, zlib
import numpy as np
sys.path.insert(0, sys.argv[1])
from parflow_b200 import configs
from parflow_b200.problem import BC, BC_DIRICHLET
from parflow_b200.solver import RichardsGPU
nx, ny, nz = 127, 129, 123
n = nx * ny * nz
assert n % 2 == 1 and n > 2000000
prob = configs.box(nx=4, ny=4, nz=4, nsteps=1)
prob.nx, prob.ny, prob.nz = nx, ny, nz
rng = np.random.default_rng(5)
prob.perm = 0.01 * np.exp(rng.standard_normal(prob.shape))
prob.bc["z_lower"] = BC(BC_DIRICHLET, (45.0,), ref_patch="z_lower")
p0 = prob.hydrostatic_ic(45.0, "z_lower") + 0.1 * rng.standard_normal(prob.shape)
out = {}
for precision in ("fp64", "mixed16"):
    for graph in (1, 0):
        g = RichardsGPU(prob, precision=precision)
        g.solve_graph(graph)
        t, dt = prob.time_plan()[0]
        g.set_time(t)
        g.set_pressure(p0)
        st = g.advance(1, dt)[0]
        p1 = g.get_pressure()
        f = g.nl_function_eval(p1, p0, g.saturation(p0), dt)
        # the same function of the same bits; n terms summed in another order
        norm = float(np.sqrt(np.sum(f * f)))
        assert st.nonlin_iters > 1 and abs(norm - st.fnorm) <= n * 2.0 ** -53 * norm, (norm, st.fnorm)
        out["%s %d" % (precision, graph)] = [zlib.crc32(p1.tobytes()), st.nonlin_iters,
                                             st.lin_iters]
        g.close()
json.dump(out, open(sys.argv[2], "w"))
"""


def _run(tmp_path, name, env):
    path = str(tmp_path / (name + ".json"))
    subprocess.run([sys.executable, "-c", CHILD, ROOT, path], env=dict(os.environ, **env),
                   check=True, timeout=300)
    return json.load(open(path))


def test_forms_of_a_large_step(tmp_path):
    import torch

    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    ref = _run(tmp_path, "default", {})
    for precision in ("fp64", "mixed16"):
        assert ref[precision + " 1"] == ref[precision + " 0"]
    assert _run(tmp_path, "gather", {"PFGPU_RESIDUAL_FACE_ONCE": "0"}) == ref
    assert _run(tmp_path, "fused", {"PFGPU_FUSE_CELLS": "100000000"}) == ref
