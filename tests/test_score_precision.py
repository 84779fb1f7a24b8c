"""Scores whose sums are small: a model whose every change is improbable (predictors
from -10 to -70), one where only some alters' changes are, and gwdsp, whose largest
possible statistic is far above those that occur. Against the CPU oracle's float64
sums: identical trajectories, scores within one float32 ulp, as
tests/test_gpu_parity.py states and derives."""
import numpy as np
import pytest

from cusna_gb300 import effects as E
from cusna_gb300 import workloads as WL
from tests.golden.make_golden import run_case
from tests.test_gpu_parity import GpuEngine, assert_parity

pytestmark = pytest.mark.gpu


def _case(n, effs, theta, x0, seed, M=2, lam=5.0):
    return dict(inp=WL.period_inputs(x0, effs), M=M, seed=seed, lam=lam, lamb=0.0, thetab=None,
                theta=np.asarray(theta, dtype=np.float64))


def _check(port, c, tag):
    ref = run_case(port, c)
    for opts in (dict(specialise=-1, warps_per_chain=1, chains_per_cta=2),
                 dict(specialise=1, warps_per_chain=4, chains_per_cta=1)):
        assert_parity(run_case(GpuEngine(**opts), c), ref, f"{tag}/{opts}")


@pytest.mark.parametrize("n", [20, 70])
@pytest.mark.parametrize("density", [-10.0, -15.0, -20.0, -24.0, -29.0, -35.0, -52.0, -58.5, -70.0])
def test_improbable_changes(gpu_lib, port, n, density):
    cov = np.round(np.random.Generator(np.random.PCG64(n)).standard_normal(n), 3)
    effs = [E.make_effect_spec("density"), E.make_effect_spec("recip"),
            E.make_effect_spec("altX", cov), E.make_effect_spec("simX", cov)]
    c = _case(n, effs, [density, 0.5, 0.3, 0.4], np.zeros((n, n), np.uint8), n + int(-10 * density))
    _check(port, c, f"n={n}/density={density}")


@pytest.mark.parametrize("n", [20, 45, 97])
@pytest.mark.parametrize("same", [-9.0, -14.0, -22.0, -31.0, -47.0, -64.0])
def test_improbable_changes_beside_probable_ones(gpu_lib, port, n, same):
    """Creating a tie within a group is improbable by one step or two; the statistics of
    those effects are 0 at every probable alter."""
    r = np.random.Generator(np.random.PCG64(7))
    half = (r.random(n) < 0.5).astype(np.float64)
    third = (np.arange(n) % 3 == 0).astype(np.float64)
    effs = [E.make_effect_spec("density"), E.make_effect_spec("recip"),
            E.make_effect_spec("sameX", half), E.make_effect_spec("sameX", third),
            E.make_effect_spec("transTrip")]
    x0 = WL.bernoulli_net(n, 0.1, seed=3)   # without ties within a group, whose end is certain
    x0[(half[:, None] == half) | (third[:, None] == third)] = 0
    c = _case(n, effs, [-1.5, 0.8, same, 0.45 * same, 0.1], x0, 11)
    _check(port, c, f"n={n}/same={same}")


@pytest.mark.parametrize("n,M", [(300, 1), (700, 1)])
def test_shared_partners_far_below_their_bound(gpu_lib, port, n, M):
    effs = [E.make_effect_spec(x) for x in ("density", "recip", "gwdspFF", "gwdspFB", "inPopSqrt")]
    c = _case(n, effs, [-2.2, 1.0, -0.05, -0.03, 0.1], WL.bernoulli_net(n, 3.0 / n, seed=n), n, M, 6.0)
    _check(port, c, f"n={n}")
