"""Weight gradients add the batch in row order, whole: rows without a gradient (their
targets are the network's own outputs) behind the others leave every bit of the weight
gradients as the shorter batch has them, but for the mean's factor, a power of two.
A product whose batch is cut into shares adds the same rows in another order for each
batch size and does not (and an epoch of training then ends with other parameters).
No tolerance: every operation scales exactly by a power of two."""
import numpy as np
import pytest

from tests.test_mlp import _Gpu, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(16, 64, 8), (16, 256, 8), (48, 272, 16)])
@pytest.mark.parametrize("b,B", [(192, 384), (256, 1024), (320, 1280)])
def test_rows_without_a_gradient_change_no_bit(gpu_lib, dims, b, B):
    n_in, hidden, n_out = dims
    g = _Gpu(*dims)
    p, X, T = _problem(seed=b, B=B, n_in=n_in, hidden=hidden, n_out=n_out)
    P, Xd = g.t(p), g.t(X)
    w, nb = g.work(B)
    y = g.torch.empty((B, n_out), device=g.dev)
    assert g.lib.cusna_mlp_forward(P.data_ptr(), Xd.data_ptr(), B, y.data_ptr(), w.data_ptr(), nb,
                                   n_in, hidden, n_out, None) == 0
    Td = g.t(T)
    Td[b:] = y[b:]
    grads = []
    for rows in (b, B):
        grad = g.torch.zeros(len(p), device=g.dev)
        assert g.lib.cusna_mlp_grad(P.data_ptr(), Xd.data_ptr(), Td.data_ptr(), None, rows,
                                    grad.data_ptr(), None, w.data_ptr(), nb, n_in, hidden, n_out,
                                    None) == 0
        grads.append(grad.double().cpu().numpy() * rows)
    o = 0
    for name, sz in (("W1", hidden * n_in), ("", hidden), ("W2", hidden * hidden), ("", hidden),
                     ("W3", n_out * hidden), ("", n_out)):
        if name:
            assert np.any(grads[0][o:o + sz])
            np.testing.assert_array_equal(grads[0][o:o + sz], grads[1][o:o + sz], err_msg=name)
        o += sz
