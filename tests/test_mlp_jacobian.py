"""The Jacobian kernel at the edges of its split: hidden widths whose rows do not
divide over the cluster, more inputs than one pass takes, one and several points,
and the single-CTA form for many points. It reads float32 pre-activations of the
bfloat16 forward pass, so it is compared with the oracle as tests/test_mlp.py does."""
import pytest

from tests.test_mlp import OM, _Gpu, _problem, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,n_wrt", [((16, 16, 1), 1), ((16, 48, 5), 9), ((32, 272, 16), 32),
                                        ((16, 2064, 3), 8)])
@pytest.mark.parametrize("B", [1, 3, 90])
def test_jacobian_matches_the_oracle(gpu_lib, dims, n_wrt, B):
    n_in, hidden, n_out = dims
    g = _Gpu(*dims)
    p, X, _ = _problem(seed=7, B=B, n_in=n_in, hidden=hidden, n_out=n_out)
    w, nb = g.work(B)
    y = g.torch.empty((B, n_out), device=g.dev)
    J = g.torch.full((B, n_out, n_wrt), float("nan"), device=g.dev)
    assert g.lib.cusna_mlp_jacobian(g.t(p).data_ptr(), g.t(X).data_ptr(), B, n_wrt, y.data_ptr(),
                                    J.data_ptr(), w.data_ptr(), nb, n_in, hidden, n_out, None) == 0
    assert _rel(J.double().cpu().numpy(), OM.jacobian(p, X, n_in, hidden, n_out, n_wrt)) < 2e-2
