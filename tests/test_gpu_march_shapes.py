"""The march form of the residual and the Jacobian (a warp walks 31 columns of a
row up through a chunk of planes) equals the gather form bit for bit on grids
around its strip width and chunk length, flat and with slopes, barriers and
permeabilities whose face means need the division (zero, subnormal, tiny).  The form is
chosen once per process (PFGPU_RESIDUAL_FACE_ONCE), so each runs in a child."""

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
from parflow_b200.solver import RichardsGPU
out = {}
for nx, ny, nz in ((1, 1, 2), (2, 1, 1), (30, 1, 3), (31, 2, 1), (32, 3, 8), (33, 8, 9),
                   (62, 9, 17), (63, 5, 16), (94, 2, 25)):
    for kind in ("box", "overland", "barrier", "tight"):
        if kind == "overland" and nx * ny == 1:
            continue  # (no slope field of one column)
        if kind == "overland":
            prob = configs.overland(nx=nx, ny=ny, nz=nz, nsteps=1, wt_depth=-0.05)
        else:
            prob = configs.box(nx=nx, ny=ny, nz=nz, nsteps=1)
        rng = np.random.default_rng(nx + 100 * ny + 10000 * nz)
        if kind == "barrier":
            prob.fbx, prob.fby, prob.fbz = (rng.uniform(0.05, 1.0, prob.shape) for _ in range(3))
        if kind == "tight":
            prob.perm = rng.choice([0.0, 5e-324, 1e-310, 1e-300, 1e-37, 1.0], size=prob.shape)
        p_old = prob.initial_pressure()
        p = p_old + 0.1 * rng.standard_normal(p_old.shape)
        x = rng.standard_normal(p.shape)
        for precision in ("fp64", "mixed"):
            g = RichardsGPU(prob, precision=precision)
            f = g.nl_function_eval(p, p_old, g.saturation(p_old), prob.dt)
            y = g.jacobian_matvec(p, prob.dt, x, p_old=p_old)
            assert np.isfinite(f).all() and np.isfinite(y).all()
            out["%dx%dx%d %s %s" % (nx, ny, nz, kind, precision)] = [
                zlib.crc32(f.tobytes()), zlib.crc32(y.tobytes())]
            g.close()
json.dump(out, open(sys.argv[2], "w"))
"""


def _run(tmp_path, form):
    path = str(tmp_path / (form + ".json"))
    env = dict(os.environ, PFGPU_RESIDUAL_FACE_ONCE=form)
    subprocess.run([sys.executable, "-c", CHILD, ROOT, path], env=env, check=True, timeout=600)
    return json.load(open(path))


def test_march_equals_gather(tmp_path):
    import torch

    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    march, gather = _run(tmp_path, "1"), _run(tmp_path, "0")
    assert march == gather
    assert len(march) == (9 * 4 - 1) * 2


@pytest.mark.parametrize("bottom", (False, True))
def test_paired_van_genuchten(bottom):
    """The residual of a grid of 2 million cells equals, bit for bit, that of a
    smaller grid with the same planes, at either end of an odd number of cells:
    a van Genuchten pass whose form depends on the size or pairs cells shows."""
    import numpy as np

    from parflow_b200 import configs
    from parflow_b200.solver import RichardsGPU

    nx, ny, nz, part = 127, 129, 123, 61
    rng = np.random.default_rng(7)
    p_old = -0.5 + 0.6 * rng.standard_normal((nz, ny, nx))
    p = p_old + 0.1 * rng.standard_normal(p_old.shape)
    perm = rng.uniform(0.01, 1.0, p.shape)
    f = []
    for planes in (slice(0, nz), slice(0, part) if bottom else slice(nz - part, nz)):
        n = planes.stop - planes.start
        prob = configs.box(nx=nx, ny=ny, nz=n, nsteps=1)
        prob.perm = perm[planes]
        g = RichardsGPU(prob, precision="fp64")
        f.append(g.nl_function_eval(p[planes], p_old[planes], g.saturation(p_old[planes]), prob.dt))
        g.close()
    assert nx * ny * nz > 2000000 > nx * ny * part and nx * ny * nz % 2 == 1
    # (the cut plane has another neighbour or a boundary)
    same = slice(0, part - 1) if bottom else slice(nz - part + 1, nz)
    np.testing.assert_array_equal(f[0][same], f[1][:-1] if bottom else f[1][1:])
