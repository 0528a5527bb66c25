"""pfgpu_time_kernel times the kernels at a state the caller gave: after
pfgpu_pc_setup alone at that call's pressure, not at the zero of the handle's
creation, where the van Genuchten pass has no logarithm to take."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["residual", "jacobian"])
def test_times_the_pressure_that_was_given(kernel):
    import torch

    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from parflow_b200 import configs
    from parflow_b200.solver import RichardsGPU

    prob = configs.box(nx=4, ny=4, nz=4, nsteps=1)
    prob.nx, prob.ny, prob.nz = 384, 384, 24
    prob.perm = np.full(prob.shape, 0.01)
    dry = -0.5 - np.random.default_rng(1).random(prob.shape)

    def best(set_pressure, p):
        g = RichardsGPU(prob)
        if set_pressure:
            g.nl_function_eval(p, p, g.saturation(p), 0.05)
            g.set_pressure(p)
        g.pc_setup(p, 0.05, p_old=p)
        g.time_kernel(kernel, 5)
        ms = min(g.time_kernel(kernel, 20)[0] for _ in range(4))
        g.close()
        return ms

    saturated, given, setup_only = best(True, -dry), best(True, dry), best(False, dry)
    # (what the pass costs: the two could not be told apart otherwise)
    assert saturated < 0.9 * given
    # the two runs of one state differ by a few percent at most, by 14 at zero pressure
    assert abs(setup_only - given) < 0.08 * given
