"""The largest networks that the no-allocation entry point's rule accepts: a chain's slice
is a little larger than the rule's accounting, and the out-rows then go to scratch. Same
results as the allocating call (as tests/test_gpu_parity.py states and derives)."""
import ctypes as C

import numpy as np
import pytest

from cusna_gb300 import effects as E
from cusna_gb300 import workloads as WL
from cusna_gb300.abi import OK
from cusna_gb300.glue import marshal_period
from tests.golden.make_golden import run_case
from tests.test_gpu_parity import GpuEngine, assert_parity
from tests.test_zz_no_alloc import _outputs, _to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,M", [(1240, 3), (1251, 40), (1260, 3)])
def test_static_entry_point_at_the_rule_s_edge(gpu_lib, n, M):
    torch = pytest.importorskip("torch")
    names = ("density", "recip") + 11 * ("inPop", "cycle3")
    effs = [E.make_effect_spec(x) for x in names]
    theta = np.array([-3.0, 1.0] + 11 * [0.002, -0.003])
    c = dict(inp=WL.period_inputs(WL.bernoulli_net(n, 3.0 / n, seed=n), effs, conditional=1, target_dist=30),
             M=M, seed=n, lam=1.0, lamb=0.0, thetab=None, theta=theta)
    ref = run_case(GpuEngine(), c)
    m = marshal_period(c["inp"], M, c["seed"], c["lam"], theta, want_ends=True)
    dev = _to_device(m, torch)
    st = gpu_lib.cusna_saom_simulate_period_static(C.byref(m.problem), C.byref(m.result), None)
    assert st == OK, gpu_lib.cusna_last_error()
    torch.cuda.synchronize()
    assert_parity(_outputs(m, dev), ref, f"n={n}")
