"""Interactions of count effects, whose bounds (two-paths times degrees) are far above
what networks hold: parameters on both sides of the largest that an interaction's
fixed-point scale once held (theta = 2^-5 for two-paths x indegrees at n = 300, 2^-4
for the same with reciprocity at n = 65), in the library's and the specialised kernel,
against the CPU oracle: identical trajectories, scores within one float32 ulp, as
tests/test_gpu_parity.py states and derives."""
import numpy as np
import pytest

from cusna_gb300 import effects as E
from cusna_gb300 import workloads as WL
from tests.golden.make_golden import run_case
from tests.test_gpu_parity import GpuEngine, assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("specialise", [-1, 1])
@pytest.mark.parametrize("n,members,thetas", [
    (300, (2, 3), (0.031, 0.032, 0.05, -0.05)),
    (65, (1, 2, 3), (0.062, 0.063, 0.1, -0.2)),
    (65, (2, 3), (0.49, 0.52, -0.9)),
    (300, (1, 2, 3), (0.0038, 0.0041, 0.03, -0.03)),
])
def test_interactions_of_counts_match_the_oracle(gpu_lib, port, n, members, thetas, specialise):
    effs = [E.make_effect_spec(x) for x in ("density", "recip", "transTrip", "inPop")]
    effs.append(E.make_interaction_spec(list(members)))
    x0 = WL.bernoulli_net(n, 6.0 / n, seed=n)
    for q, t in enumerate(thetas):
        c = dict(inp=WL.period_inputs(x0, effs), M=2, seed=100 * n + q, lam=4.0, lamb=0.0, thetab=None,
                 theta=np.array([-2.5, 0.9, 0.05, -0.02, t]))
        got = run_case(GpuEngine(specialise=specialise), c)
        assert_parity(got, run_case(port, c), f"n={n}/{members}/theta={t}")
