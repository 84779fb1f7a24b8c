"""Count matrices are optional: under a cap on their memory that none fits, and where the
device has not the memory free, simulations, plans and multi-network calls run with
popcounts and give the same bits. A batch with networks on both sides of twelve
32-actor words gives each problem its own call's bits."""
import numpy as np
import pytest

from cusna_gb300 import sim as G
from cusna_gb300 import workloads as WL
from cusna_gb300.glue import marshal_multi, marshal_period
from tests.golden.make_golden import run_case
from tests.test_gpu_parity import GpuEngine

pytestmark = pytest.mark.gpu


def _same(a, b, tag):
    assert set(a) == set(b)
    for key in a:
        np.testing.assert_array_equal(a[key], b[key], err_msg=f"{tag}:{key}")


def _marshal(c):
    return marshal_period(c["inp"], c["M"], c["seed"], c["lam"], c["theta"], lamb=c["lamb"],
                          thetab=c["thetab"], want_ends=True)


@pytest.mark.parametrize("cap", ["0", "1"])
def test_a_cap_on_the_matrices(gpu_lib, monkeypatch, cap):
    c = WL.parity_case("structural", seed=4, n=360, M=12)
    inp, seed, lam, th = WL.multi_case("cross", seed=3, n=355, M=6)
    runs = []
    for value in (None, cap):
        if value is not None:
            monkeypatch.setenv("CUSNA_COUNTS_MAX_MB", value)
        plan = G.SimPlan([_marshal(c)])
        plan.launch()
        runs.append((run_case(GpuEngine(specialise=-1), c), run_case(GpuEngine(specialise=1), c),
                     plan.outputs()[0], G.simulate_multi(marshal_multi(inp, 6, seed, lam, th))))
        plan.close()
    for q, (a, b) in enumerate(zip(*runs)):
        _same(a, b, f"call {q}")


def test_a_device_without_the_memory(gpu_lib):
    torch = pytest.importorskip("torch")
    inp, M, seed, lam, theta, lamb, thetab = WL.c4_period(M=1024)
    inp.conditional, inp.target_dist = 1, 5
    args = (inp, M, seed, lam, theta)
    with_room = G.simulate(marshal_period(*args, lamb=lamb, thetab=thetab))

    def call():   # another thread has another arena
        out.append(G.simulate(marshal_period(*args, lamb=lamb, thetab=thetab)))
    import threading
    out = []
    torch.cuda.empty_cache()
    hog = torch.empty(max(torch.cuda.mem_get_info()[0] - (3 << 29), 1), dtype=torch.uint8, device="cuda")
    try:
        t = threading.Thread(target=call)
        t.start()
        t.join()
    finally:
        del hog
        torch.cuda.empty_cache()
    _same(out[0], with_room, "without the memory")


def test_a_batch_on_both_sides_of_the_rule(gpu_lib):
    cases = [WL.parity_case(k, seed=q, n=n, M=m) for q, (k, n, m) in enumerate(
        (("structural", 353, 3), ("structural", 60, 5), ("structural", 352, 2), ("structural", 400, 4)))]
    batch = G.simulate_batch([_marshal(c) for c in cases])
    plan = G.SimPlan([_marshal(c) for c in cases])
    plan.launch()
    planned = plan.outputs()
    plan.close()
    for q, c in enumerate(cases):
        one = run_case(GpuEngine(specialise=-1), c)
        _same(batch[q], one, f"batch {q}")
        _same(planned[q], one, f"plan {q}")
