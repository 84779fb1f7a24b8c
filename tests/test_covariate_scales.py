"""Covariates so small or so large that their power of two has no fixed-point scale (and
products that underflow): the chain runs in float64, as the CPU oracle (identical
trajectories, scores within one float32 ulp, as tests/test_gpu_parity.py states)."""
import numpy as np
import pytest

from cusna_gb300 import effects as E
from cusna_gb300 import workloads as WL
from tests.golden.make_golden import run_case
from tests.test_gpu_parity import GpuEngine, assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("specialise", [-1, 1])
@pytest.mark.parametrize("scale,theta", [(1e-305, 1e30), (1e-295, 0.4), (1e-120, 0.3), (1e270, 1e-30), (1e301, 0.0)])
def test_covariates_beyond_the_scales(gpu_lib, port, scale, theta, specialise):
    n = 30
    cov = np.round(np.random.Generator(np.random.PCG64(3)).standard_normal(n), 3)
    effs = [E.make_effect_spec("density"), E.make_effect_spec("recip"), E.make_effect_spec("egoX", cov),
            E.make_effect_spec("altX", cov), E.make_interaction_spec([2, 3])]
    inp = WL.period_inputs(WL.bernoulli_net(n, 0.1, seed=4), effs)
    inp.vmat = np.asarray(inp.vmat, dtype=np.float64) * scale
    c = dict(inp=inp, M=3, seed=5, lam=5.0, lamb=0.0, thetab=None,
             theta=np.array([-2.0, 0.9, theta, -theta, 0.0]))
    assert_parity(run_case(GpuEngine(specialise=specialise), c), run_case(port, c), f"{scale}/{theta}")
