"""Chains whose ministeps hand their score sums' scaling on: dense networks with large
predictors, where an actor's largest weight needs a scaling and the next actor's may
not. Every team size and both kernels give the same bits, and the CPU oracle's
trajectories with scores within one float32 ulp (tests/test_gpu_parity.py states and
derives); two networks of a chain hand on a scaling each."""
import numpy as np
import pytest

from cusna_gb300 import effects as E
from cusna_gb300 import sim as G
from cusna_gb300 import workloads as WL
from cusna_gb300.glue import marshal_multi
from tests.golden.make_golden import run_case
from tests.test_gpu_parity import GpuEngine, assert_parity
from tests.test_multi import assert_multi_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,density", [(40, 0.3), (150, 0.12), (360, 0.1)])
def test_dense_networks_match_the_oracle_for_every_team(gpu_lib, port, n, density):
    cov = (np.random.Generator(np.random.PCG64(n)).random(n) < 0.5).astype(np.float64)
    effs = [E.make_effect_spec(x) for x in ("density", "recip", "transTrip", "outTrunc")]
    effs += [E.make_effect_spec("sameX", cov), E.make_effect_spec("altX", cov)]
    c = dict(inp=WL.period_inputs(WL.bernoulli_net(n, density, seed=n), effs), M=3, seed=n, lam=6.0,
             lamb=0.0, thetab=None, theta=np.array([-2.4, 1.9, 0.35, 0.1, 0.45, 0.2]))
    ref = run_case(GpuEngine(specialise=-1, warps_per_chain=1, chains_per_cta=2), c)
    assert_parity(ref, run_case(port, c), f"n={n}")
    for opts in (dict(specialise=-1, warps_per_chain=4, chains_per_cta=1),
                 dict(specialise=1, warps_per_chain=1, chains_per_cta=4),
                 dict(specialise=1, warps_per_chain=8, chains_per_cta=1)):
        got = run_case(GpuEngine(**opts), c)
        for key in ref:
            np.testing.assert_array_equal(got[key], ref[key], err_msg=f"n={n}/{opts}/{key}")


def test_two_dense_networks_match_the_oracle(gpu_lib, port):
    inp, seed, lam, th = WL.multi_case("cross", seed=5, n=60, M=3)
    r = np.random.Generator(np.random.PCG64(5))
    for q, x in enumerate(inp.x0s):
        inp.x0s[q] = (x | (r.random(x.shape) < 0.2 * (1 + q))).astype(np.uint8)
        np.fill_diagonal(inp.x0s[q], 0)
    ref = port.simulate_multi(marshal_multi(inp, 3, seed, lam, 1.5 * th))
    for mode in (0, 2):
        G.specialise_mode(mode)
        try:
            got = G.simulate_multi(marshal_multi(inp, 3, seed, lam, 1.5 * th))
        finally:
            G.specialise_mode(-1)
        assert_multi_parity(got, ref, f"specialise={mode}")
