"""The network's one-launch inference against the layer-by-layer kernels that training runs, at
the edges of its tiles (input widths around a K slice, outputs around a padded tile, the smallest
and largest widths, depths on both sides of its layer limit). Both take the same products in the
same order with the same rounding points, so the outputs are equal bit for bit: the mean-square
loss of the training forward against the inference outputs as targets is exactly zero. The
weight gradients' slices: batches of one slice, of an odd number and of many, against the oracle
(2e-2 relative per layer, as the gradient test of the same kernels)."""
import numpy as np
import pytest

from casim_b200 import surrogate as sg
from oracle import mlp_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,n_out,width,depth,rows", [(1, 1, 128, 1, 128), (63, 20, 256, 4, 384), (64, 128, 128, 2, 128),
                                                         (65, 129, 256, 3, 256), (256, 256, 256, 2, 128), (7, 5, 128, 15, 128),
                                                         (7, 5, 128, 16, 128), (63, 20, 256, 4, 148 * 128 + 128)])
def test_inference_equals_training_forward(cuda_device, n_in, n_out, width, depth, rows):
    import torch
    net = sg.Surrogate(n_in, n_out, width=width, depth=depth, seed=n_in + n_out)
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn((rows, n_in), generator=g, device="cuda")
    y = net.forward(x)
    assert torch.isfinite(y).all() and float(y.abs().max()) > 0
    loss, _ = net.gradients(x, y)
    assert loss == 0.0
    net.close()


@pytest.mark.parametrize("rows", [128, 384, 4096 + 128])
def test_sliced_weight_gradients_match_oracle(cuda_device, rows):
    import torch
    n_in, n_out = 40, 20
    net = sg.Surrogate(n_in, n_out, width=128, depth=2, seed=9)
    rng = np.random.default_rng(rows)
    x = rng.uniform(-1, 1, size=(rows, n_in)).astype(np.float32)
    t = rng.normal(size=(rows, n_out)).astype(np.float32)
    for r in (rows, 128):  # then a smaller batch in the same workspaces
        loss, g = net.gradients(torch.from_numpy(x[:r]).cuda(), torch.from_numpy(t[:r]).cuda())
        ref_loss, ref = mlp_oracle.gradients(net.unflatten(net.get_params()), x[:r], t[:r], n_in, n_out)
        assert abs(loss - ref_loss) <= 1e-3 * abs(ref_loss)
        for l, ((gw, gb), (rw, rb)) in enumerate(zip(net.unflatten(g), ref)):
            assert np.linalg.norm(gw - rw) <= 2e-2 * np.linalg.norm(rw), (r, l)
            assert np.linalg.norm(gb - rb) <= 2e-2 * max(np.linalg.norm(rb), 1e-30), (r, l)
    net.close()
