"""Large sparse networks and products of counts, whose statistics' bounds from the
number of actors alone leave the fixed-point range: the degrees that occur decide.
Against the CPU oracle (identical trajectories, scores within one float32 ulp, as
tests/test_gpu_parity.py states and derives), with networks that outgrow the bound a
chain starts with, and in time: parameters that the bounds of n would refuse cost at
most twice those that they allow (in float64 every ministep costs several times as
much)."""
import numpy as np
import pytest

from cusna_gb300 import effects as E
from cusna_gb300 import sim as G
from cusna_gb300 import workloads as WL
from cusna_gb300.glue import marshal_period
from tests.golden.make_golden import run_case
from tests.test_gpu_parity import GpuEngine, assert_parity

pytestmark = pytest.mark.gpu


def _case(n, names, theta, x0, seed, M=2, **kw):
    effs = [E.make_interaction_spec(list(x)) if isinstance(x, tuple) else E.make_effect_spec(x)
            for x in names]
    return dict(inp=WL.period_inputs(x0, effs, **kw), M=M, seed=seed, lam=1.0, lamb=0.0, thetab=None,
                theta=np.array(theta))


@pytest.mark.parametrize("specialise", [-1, 1])
def test_products_of_counts_beyond_the_bounds_of_n(gpu_lib, port, specialise):
    for n, t in ((300, 0.1), (300, -0.3), (65, 2.5)):
        c = _case(n, ("density", "recip", "transTrip", "inPop", (2, 3)), [-2.5, 0.9, 0.05, -0.02, t],
                  WL.bernoulli_net(n, 5.0 / n, seed=n), n, conditional=1, target_dist=4 * n)
        assert_parity(run_case(GpuEngine(specialise=specialise), c), run_case(port, c), f"n={n}/{t}")


@pytest.mark.parametrize("warps,per_cta", [(1, 2), (4, 1)])
def test_large_parameters_match_the_oracle(gpu_lib, port, warps, per_cta):
    n = 1100
    c = _case(n, ("density", "recip", "transTrip", "cycle3", "inPop", "outTrunc"),
              [-4.5, 2.0, 6.0, -3.0, -1.0, 0.5], WL.bernoulli_net(n, 2.0 / n, seed=3), 5, M=1,
              conditional=1, target_dist=60)
    opts = dict(warps_per_chain=warps, chains_per_cta=per_cta)
    assert_parity(run_case(GpuEngine(**opts), c), run_case(port, c), str(opts))


def test_a_network_that_outgrows_its_bound(gpu_lib, port):
    """From an empty network to one of high degrees: ministeps beyond the bound run in float64."""
    n = 70
    c = _case(n, ("density", "recip", "inAct", "outAct", "outPop", (3, 4)),
              [1.2, 0.1, -0.02, 0.01, 0.02, 2.6], np.zeros((n, n), np.uint8), 9, M=2, conditional=1,
              target_dist=900)
    c["theta"][5] = 2.6
    ref = run_case(port, c)
    for opts in (dict(specialise=-1, warps_per_chain=1, chains_per_cta=2),
                 dict(specialise=1, warps_per_chain=2, chains_per_cta=1)):
        assert_parity(run_case(GpuEngine(**opts), c), ref, str(opts))


def test_no_cliff_at_the_bounds_of_n(gpu_lib):
    n, ms = 2000, []
    x0 = WL.bernoulli_net(n, 3.0 / n, seed=2)
    # the same model twice: one effect's parameter, and two that add up to it
    effs = [E.make_effect_spec(x) for x in ("density", "recip", "transTrip", "transTrip", "inPop")]
    for theta in ([-3.5, 1.0, 0.5, 0.0, 0.05], [-3.5, 1.0, 3.5, -3.0, 0.05]):
        inp = WL.period_inputs(x0, effs, conditional=1, target_dist=800)
        m = marshal_period(inp, 152, 3, 1.0, np.array(theta))
        best = float("inf")
        for _ in range(3):
            o = G.options(specialise=1, warps_per_chain=4, chains_per_cta=1)
            out = G.simulate_ex(m, o)
            best = min(best, o.elapsed_ms / out["steps"].max())
        ms.append(best)
    assert ms[1] < 2.0 * ms[0], ms
