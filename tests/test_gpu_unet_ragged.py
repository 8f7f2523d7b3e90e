"""The network's kernels at shapes where their tiles end (the input layer's
weight gradient, the bias gradients, decoder convolutions that read the skip
connection in place), against the numpy oracle, with the tolerances that
test_gpu_unet.py derives for it: 1e-2 for the output, 5e-2 for each layer's
gradient."""
import pytest

from oracle import unet_oracle as U
from flowlab_gb300 import native
from tests.test_gpu_unet import batch, random_params, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(1, 8, 8), (2, 24, 40), (3, 16, 136), (1, 72, 264)])
def test_ragged_shapes_match_oracle(B, H, W):
    th = random_params(21)
    x, t, m = batch(22, B=B, H=H, W=W)
    net = native.Unet(B * H * W)
    try:
        net.set_params(th)
        out = net.forward(x)
        loss, g = net.train_step(x, t, m, update=False, want_grad=True)
    finally:
        net.close()
    ref_net = U.Net(th, bf16=True)
    assert rel(out, ref_net.forward(x)) < 1e-2
    ref_loss, dout, _ = U.loss_and_grad(ref_net, x, t, m)
    ref = ref_net.backward(dout)
    assert abs(loss - ref_loss) <= 1e-2 * ref_loss
    layout, _ = U.param_layout()
    for name, wo, nw, bo, cout in layout:
        assert rel(g[wo:wo + nw], ref[wo:wo + nw]) < 5e-2, (name, rel(g[wo:wo + nw], ref[wo:wo + nw]))
        assert rel(g[bo:bo + cout], ref[bo:bo + cout]) < 5e-2, name
