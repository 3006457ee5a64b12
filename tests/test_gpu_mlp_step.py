"""GPU checks of the fused training step: batches of one tile, of ragged tiles and of more
tiles than the GPU has CTAs (a CTA then accumulates several tiles in tensor memory), against
the BF16-emulating oracle; and the fixed summation order (the same bits from run to run)."""
import numpy as np
import pytest

from higherharmonics_b200 import api
from oracle import mlp_oracle as MO
from tests.test_gpu_learned import GRAD_TOL, PRED_TOL_TC, _args, _synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [127, 129, 148 * 128 + 1, 40001])
def test_step_gradients_over_tiles(engine, n):
    rec = _synthetic(n)
    net = api.mlp_init(11, rec if n > 1000 else _synthetic(4096))
    g, loss = engine.mlp_gradients(rec, net)
    loss_ref, g_ref = MO.loss_and_grad(net.param_array(), rec, *_args(net), emulate=True)
    assert abs(loss - loss_ref) <= 1e-4 * loss_ref
    o = 0
    for name, shape in MO.LAYOUT:
        k = int(np.prod(shape))
        err = np.linalg.norm(g[o:o + k] - g_ref[o:o + k]) / np.linalg.norm(g_ref[o:o + k])
        assert err <= GRAD_TOL, (name, err)
        o += k
    pred = engine.mlp_predict(rec, net, path=1)
    assert np.max(np.abs(pred - MO.predict(net.param_array(), rec, *_args(net), emulate=True))) <= PRED_TOL_TC


def test_training_is_reproducible(engine):
    rec = _synthetic(5000)
    out = []
    for _ in range(2):
        net = api.mlp_init(2, rec)
        loss, _ = engine.mlp_train(rec, net, api.train_opts(epochs=3, batch=384))
        out.append((net.param_array().copy(), loss.copy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
