"""Behaviour ministeps at the edges of the warp's split: more than 32 neighbours,
and more than 32 words of row. Outputs as tests/test_gpu_parity.py compares them
(the sums keep the reference's order)."""
import pytest

from cusna_gb300 import workloads as WL
from tests.golden.make_golden import run_case
from tests.test_gpu_parity import GpuEngine, assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lam", [(31, 4.0), (420, 1.0), (1056, 0.1)])
def test_behaviour_steps_match_the_oracle(gpu_lib, port, n, lam):
    c = WL.parity_case("coevol", seed=6, n=n, M=2)
    c["lam"], c["lamb"] = lam, 2.0 * lam
    assert_parity(run_case(GpuEngine(), c), run_case(port, c), f"coevol/n={n}")
