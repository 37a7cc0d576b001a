"""The warm-start network against the CPU oracle where the tiles of its
predictions and of its training products end: 64 rows and 64 outputs a head
tile, rank 64, 32 x 16 hidden tiles, word loads only for even sizes."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_warmstart import _fp, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,batch", [((1, 1, 1, 1), 1), ((32, 64, 64, 130), 63), ((32, 64, 64, 128), 64),
                                        ((32, 66, 64, 127), 64), ((31, 65, 63, 190), 64), ((32, 64, 64, 64), 65),
                                        ((32, 64, 65, 64), 64), ((16, 512, 64, 9601), 33), ((16, 48, 62, 9602), 128),
                                        ((16, 48, 64, 300), 129)])
def test_loss_gradient_and_prediction(lib, dims, batch):
    """Loss to 1e-5, each gradient block to 2e-4 and outputs to 1e-4 of their
    largest entry: products of BF16 weights with FP32 values in three BF16
    parts are exact to 2^-24, gradients of pairs to 2^-16, each times the
    square root of the terms of a sum."""
    mo = _oracle()
    rng = np.random.default_rng(sum(dims) + batch)
    fp = C.POINTER(C.c_float)
    net = lib.pdhcg_b200_mlp_create(*dims, 7)
    try:
        w = (rng.standard_normal(lib.pdhcg_b200_mlp_num_params(net)) * 0.3).astype(np.float32)
        assert lib.pdhcg_b200_mlp_set_params(net, _fp(w)) == 0
        x, t = (rng.standard_normal((batch, d)).astype(np.float32) for d in (dims[0], dims[3]))
        tl = rng.standard_normal(batch).astype(np.float32)
        loss, g = C.c_double(), np.zeros(w.size, np.float32)
        assert lib.pdhcg_b200_mlp_loss_grad(net, batch, _fp(x), _fp(t), _fp(tl), C.byref(loss),
                                            g.ctypes.data_as(fp)) == 0
        lo, go, oo, lwo = mo.loss_grad(w.astype(np.float64), x.astype(np.float64), t, tl, *dims)
        assert abs(loss.value - lo) <= 1e-5 * abs(lo)
        o = 0
        for sh in mo.shapes(*dims):
            k = int(np.prod(sh))
            np.testing.assert_allclose(g[o:o + k], go[o:o + k], rtol=0, atol=2e-4 * max(np.abs(go[o:o + k]).max(), 1e-12))
            o += k
        out, lw = np.zeros((batch, dims[3]), np.float32), np.zeros(batch, np.float32)
        assert lib.pdhcg_b200_mlp_predict(net, batch, _fp(x), out.ctypes.data_as(fp), lw.ctypes.data_as(fp)) == 0
        np.testing.assert_allclose(out, oo, rtol=0, atol=1e-4 * np.abs(oo).max())
        np.testing.assert_allclose(lw, lwo, rtol=0, atol=1e-4 * np.abs(lwo).max())
        # one training step moves every parameter against its gradient by lr m / (sqrt(v) + eps)
        # = lr g / (|g| + eps)
        la = C.c_double()
        assert lib.pdhcg_b200_mlp_train(net, batch, _fp(x), _fp(t), _fp(tl), 1, batch, 1e-3, C.byref(la)) == 0
        w1 = np.zeros_like(w)
        assert lib.pdhcg_b200_mlp_get_params(net, w1.ctypes.data_as(fp)) == 0
        big = np.abs(g) > 1e-3 * np.abs(g).max()
        np.testing.assert_allclose((w1 - w)[big], -1e-3 * np.sign(g[big]), rtol=0, atol=1e-5)
    finally:
        lib.pdhcg_b200_mlp_free(net)
