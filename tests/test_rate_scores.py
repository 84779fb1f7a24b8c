"""Scores of out- and in-degree rate effects, which read the focal actor's degrees after
the ministep's toggle, for teams of one and several warps, directed and symmetric
networks, with and without the statistics (whose code orders the end of a chain),
against the CPU oracle as tests/test_gpu_parity.py states and derives."""
import numpy as np
import pytest

from cusna_gb300 import sim as G
from cusna_gb300 import workloads as WL
from cusna_gb300.glue import marshal_period
from tests.test_gpu_parity import assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["baseline", "symmetric"])
@pytest.mark.parametrize("n", [20, 65])
@pytest.mark.parametrize("warps,per_cta", [(1, 1), (1, 4), (2, 2), (4, 1)])
def test_degree_rate_scores_match_the_oracle(gpu_lib, port, kind, n, warps, per_cta):
    c = WL.parity_case(kind, seed=n, n=n, M=6)
    c["inp"].rkind = np.array([1, 2], dtype=np.int32)
    c["inp"].ralpha = np.array([0.05, -0.04], dtype=np.float32)
    c["inp"].ru = np.zeros((2, n), dtype=np.float32)
    args = (c["inp"], c["M"], c["seed"], c["lam"], c["theta"])
    ref = port.simulate(marshal_period(*args))
    assert ref["rscores"].any()
    opts = dict(warps_per_chain=warps, chains_per_cta=per_cta)
    for drop in ((), ("stats",)):
        m = marshal_period(*args)
        m.drop_outputs(drop)
        got = G.simulate_ex(m, G.options(**opts))
        assert_parity(got, {k: v for k, v in ref.items() if k in got}, f"{kind}/n={n}/{opts}/{drop}")
