"""Two-path counts kept as matrices (networks of twelve and more 32-actor words):
simulations across the rule's edge against the CPU oracle, for every counter
that a model reads, symmetric networks (paired toggles), masks and composition,
and two networks that read each other. Trajectories and integer outputs are
identical, scores within one float32 ulp, as tests/test_gpu_parity.py states
and derives."""
import pytest

from cusna_gb300 import sim as G
from cusna_gb300 import workloads as WL
from cusna_gb300.glue import marshal_multi
from tests.golden.make_golden import run_case
from tests.test_gpu_parity import GpuEngine, assert_parity
from tests.test_multi import assert_multi_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [352, 353, 385])
@pytest.mark.parametrize("kind", ["structural", "gw", "symmetric", "masks", "composition"])
def test_matrices_match_the_oracle(gpu_lib, port, kind, n):
    c = WL.parity_case(kind, seed=n, n=n, M=2)
    ref = run_case(port, c)
    assert_parity(run_case(GpuEngine(), c), ref, f"{kind}/n={n}")
    for warps, per_cta in ((1, 4), (4, 1)):   # one and several warps share the updates
        got = run_case(GpuEngine(warps_per_chain=warps, chains_per_cta=per_cta), c)
        assert_parity(got, ref, f"{kind}/n={n}/warps={warps}")


@pytest.mark.parametrize("specialise", [0, 2])
@pytest.mark.parametrize("kind", ["cross", "symmetric"])
def test_matrices_of_two_networks_match_the_oracle(gpu_lib, port, kind, specialise):
    inp, seed, lam, th = WL.multi_case(kind, seed=3, n=355, M=2)
    ref = port.simulate_multi(marshal_multi(inp, 2, seed, lam, th))
    G.specialise_mode(specialise)
    try:
        got = G.simulate_multi(marshal_multi(inp, 2, seed, lam, th))
    finally:
        G.specialise_mode(-1)
    assert_multi_parity(got, ref, kind)
