"""Start networks with self-ties (the C ABI accepts them) under transTies, whose masks then
hold the focal actor itself: by popcounts (n = 352) and by count matrices (n = 353),
against the CPU oracle as tests/test_gpu_parity.py states and derives."""
import numpy as np
import pytest

from cusna_gb300 import effects as E
from cusna_gb300 import workloads as WL
from tests.golden.make_golden import run_case
from tests.test_gpu_parity import GpuEngine, assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("specialise", [-1, 1])
@pytest.mark.parametrize("n", [352, 353])
def test_self_ties_under_transties(gpu_lib, port, n, specialise):
    x0 = WL.bernoulli_net(n, 2.5 / n, seed=n)
    x0[np.arange(0, n, 2), np.arange(0, n, 2)] = 1
    effs = [E.make_effect_spec(x) for x in ("density", "recip", "transTies", "transTrip")]
    c = dict(inp=WL.period_inputs(x0, effs), M=3, seed=n, lam=6.0, lamb=0.0, thetab=None,
             theta=np.array([-2.3, 1.0, 1.5, 0.1]))
    assert c["inp"].x0.diagonal().any()
    assert_parity(run_case(GpuEngine(specialise=specialise), c), run_case(port, c), f"n={n}")
