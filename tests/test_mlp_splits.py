"""Weight gradients whose K (the batch) is split over a cluster: one chunk of 64
rows (no split), an even split, a share that is empty, ragged last chunks, and
products with several tiles. Tolerances as tests/test_mlp.py states for the same
products (bfloat16 operands, float32 sums whose order does not matter at 2e-3)."""
import numpy as np
import pytest

from tests.test_mlp import OM, _Gpu, _problem, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(16, 256, 8), (16, 16, 1), (48, 272, 16)])
@pytest.mark.parametrize("B", [16, 192, 320, 1040])
def test_split_weight_gradients_match_the_oracle(gpu_lib, dims, B):
    n_in, hidden, n_out = dims
    g = _Gpu(*dims)
    p, X, T = _problem(seed=B, B=B, n_in=n_in, hidden=hidden, n_out=n_out)
    w, nb = g.work(B)
    grads = []
    for _ in range(2):
        grad = g.torch.zeros(len(p), device=g.dev)
        loss = g.torch.zeros(1, device=g.dev)
        assert g.lib.cusna_mlp_grad(g.t(p).data_ptr(), g.t(X).data_ptr(), g.t(T).data_ptr(), None, B,
                                    grad.data_ptr(), loss.data_ptr(), w.data_ptr(), nb, n_in, hidden,
                                    n_out, None) == 0
        grads.append(grad.double().cpu().numpy())
    np.testing.assert_array_equal(grads[0], grads[1])
    _, g_bf = OM.loss_grad(p, X, T, n_in, hidden, n_out, bf16=True)
    o = 0
    for sz in (hidden * n_in, hidden, hidden * hidden, hidden, n_out * hidden, n_out):
        assert _rel(grads[0][o:o + sz], g_bf[o:o + sz]) < 5e-3
        o += sz
