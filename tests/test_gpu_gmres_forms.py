"""The one-launch Gram-Schmidt step of short vectors (a cluster of up to eight
blocks, vectors of up to 65536 cells) against the general path, on vectors
around the sizes where it takes another block.  The path is chosen once per
process (PFGPU_MGS_CELLS), so each runs in a child."""

import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHAPES = ((1, 1, 3), (7, 5, 3), (16, 16, 8), (41, 10, 5), (32, 16, 8), (17, 61, 4), (32, 32, 8),
          (91, 9, 11), (64, 32, 32), (99, 31, 22))

CHILD = r"""
import json, sys
sys.path.insert(0, sys.argv[1])
from parflow_b200 import configs
from parflow_b200.solver import RichardsGPU
out = {}
for nx, ny, nz in json.loads(sys.argv[3]):
    for graph in (0, 1):
        prob = configs.box(nx=nx, ny=ny, nz=nz, nsteps=2)
        g = RichardsGPU(prob)
        g.solve_graph(graph)
        ps, sts = g.run()
        out["%d %d %d %d" % (nx, ny, nz, graph)] = [
            [int(s.nonlin_iters) for s in sts], [int(s.lin_iters) for s in sts],
            ps[-1].ravel().tolist()]
        g.close()
json.dump(out, open(sys.argv[2], "w"))
"""


def _run(tmp_path, cells):
    path = str(tmp_path / (cells + ".json"))
    env = dict(os.environ, PFGPU_MGS_CELLS=cells)
    subprocess.run([sys.executable, "-c", CHILD, ROOT, path, json.dumps(SHAPES)], env=env,
                   check=True, timeout=900)
    return json.load(open(path))


def test_gram_schmidt_forms(tmp_path):
    import numpy as np
    import torch

    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    short, general = _run(tmp_path, "65536"), _run(tmp_path, "0")
    for key, (newton, linear, p) in short.items():
        assert newton == general[key][0], key
        assert linear == general[key][1], key
        # the sums differ in their order: n eps = 65536 * 2.2e-16 = 1.5e-11 of
        # each scalar at most, over some 20 Krylov vectors: 3e-10 of the heads
        want = np.array(general[key][2])
        assert np.abs(np.array(p) - want).max() <= 3e-10 * max(1.0, np.abs(want).max()), key
