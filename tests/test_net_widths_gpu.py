"""One-launch inference at the hidden widths that training's 128-row weight-gradient tiles do not
serve (64 and 192), with inputs padded to less, as much and more than the width, against the oracle's
forward pass (2e-2 of the largest output, the tolerance of the other forward test: a different FP32
summation order can flip a BF16 rounding of an activation)."""
import numpy as np
import pytest

from casim_b200 import surrogate as sg
from oracle import mlp_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,n_out,width,depth,rows", [(20, 7, 64, 1, 128), (64, 128, 64, 4, 256), (250, 20, 64, 2, 384), (63, 20, 192, 4, 256),
                                                         (180, 200, 192, 3, 128), (256, 256, 192, 16, 128)])
def test_forward_matches_oracle(cuda_device, n_in, n_out, width, depth, rows):
    import torch
    net = sg.Surrogate(n_in, n_out, width=width, depth=depth, seed=n_in)
    x = np.random.default_rng(rows + n_in).uniform(-2, 2, size=(rows, n_in)).astype(np.float32)
    y = net.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    ref, _, _ = mlp_oracle.forward(net.unflatten(net.get_params()), x, n_in)
    ref = ref[:, :n_out]
    assert np.max(np.abs(y - ref)) <= 2e-2 * np.max(np.abs(ref))
    net.close()
