"""The network's gradients layer by layer against the FP64 oracle, at sizes that run each
width of the convolution kernels in both directions and split the weight gradients into
many chunks of voxels, the last one partial."""
import numpy as np
import pytest

import homo3d_b200 as H
import oracle.warmnet_oracle as W

pytestmark = pytest.mark.gpu


# output channels per thread, forward / input gradient, over the levels: 8, 4, 2 / 8, 4, 2
# at 24^3 and 32^3, 4, 2 / 4, 2 at 16^3; 12 to 256 chunks
@pytest.mark.parametrize("R,B", [(16, 6), (24, 3), (32, 4)])
def test_gradients_per_layer(torch_cuda, R, B):
    torch = torch_cuda
    net = H.WarmNet(R, max_batch=B, seed=3)
    p = W.init_params(5).astype(np.float32)
    net.set_params(p)
    rng = np.random.default_rng(R)
    x = rng.uniform(0.0, 1.0, (B, R ** 3)).astype(np.float32)
    t = rng.standard_normal((B, W.NOUT, R ** 3)).astype(np.float32)
    p64, x64 = p.astype(np.float64), x.astype(np.float64)
    y = net.forward(torch.tensor(x, device="cuda")).cpu().numpy()
    yref = W.forward(p64, x64)
    assert np.abs(y - yref).max() <= 1e-4 * np.abs(yref).max()
    loss = net.gradients(torch.tensor(x, device="cuda"), torch.tensor(t, device="cuda"))
    lref, gref = W.loss_and_grad(p64, x64, t.astype(np.float64))
    assert abs(loss - lref) <= 1e-5 * abs(lref)
    layers = W.unpack(net.grads()), W.unpack(gref)
    for l, ((gw, gb), (rw, rb)) in enumerate(zip(*layers)):
        for a, r in ((gw, rw), (gb, rb)):
            err = np.linalg.norm(a - r) / np.linalg.norm(r)
            # a pre-activation within rounding of zero switches a ReLU: up to 1e-5 of a layer
            assert err < 1e-4, (l, err)
            # the output layer has none behind it: FP32 products and sums of its inputs,
            # themselves right to about 6e-8, with chunks added in FP64
            if l == len(layers[0]) - 1:
                assert err < 1.5e-7, err
    net.close()
