"""Parameter gradients at the edges of the gradient kernels' tiles: 32 x 8
voxel tiles of the one-channel layers, 16 x 8 x 2 of the 32-channel ones, against
the FP64 oracle with the tolerance of the full gradient test (BF16 activations)."""
import numpy as np
import pytest

from ctbb_icd_b200 import learned as L
from oracle import cnn_oracle as O
from test_gpu_cnn import FWD_TOL, GRAD_TOL, _phantom, _tensors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 3, 2), (2, 8, 32), (2, 9, 33), (3, 17, 65)])
def test_gradient_at_tile_edges(ctx, shape):
    import torch

    net = L.WarmStartNet(ctx, 1)
    p = O.init_params(1, seed=5).astype(np.float32)
    net.set_params(p)
    x = _phantom(shape, 4).astype(np.float32)
    xc = (x + 0.004 * np.cos(np.arange(x.size).reshape(shape) * 0.61)).astype(np.float32)
    loss = net.accumulate_gradient(torch.from_numpy(x).cuda(), torch.from_numpy(xc).cuda())
    g = net.gradient().astype(np.float64)
    ref_loss, ref, _ = O.loss_and_grad(p.astype(np.float64), x, xc, 1, s_in=L.S_IN, s_out=L.S_OUT)
    assert abs(loss - ref_loss) <= 2 * FWD_TOL * ref_loss
    for name, a, b in _tensors(1):
        err = np.linalg.norm(g[a:b] - ref[a:b]) / max(np.linalg.norm(ref[a:b]), 1e-30)
        assert err < GRAD_TOL, (name, err)
    net.free()
