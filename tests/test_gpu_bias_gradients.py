"""The bias gradients' rounding: a CTA of the weight-gradient kernel adds its voxels'
sum once.  N additions to a sum that grows evenly round it by ulp / sqrt(12) each,
ulp <= eps of what has been added, eps sqrt(N) / 6 = 2.4e-7 of the sum in all for
N = 152 (one CTA an SM); 3e-7 leaves the threads' own sums their share."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_level0_bias_gradients():
    import torch
    from oracle import unet_ref as U
    from vortegrid_gb300 import warmstart as ws
    edge = 128
    net, grid = ws.Network(edge), ws.field_grid(edge + 1)
    err = []
    for seed in range(4):
        net.set_params(ws.init_params(seed=seed, zero_output=False), 0.5)
        rng = np.random.default_rng(seed)
        n3 = (edge + 1) ** 3
        rhs = torch.from_numpy(rng.normal(0, 1, (n3, 3)).astype(np.float32)).cuda()
        vp = torch.from_numpy(rng.normal(0, 1e-3, (n3, 3)).astype(np.float32)).cuda()
        net.backward(grid, rhs, vp, want_loss=True)
        grads, o = net.grads(), 0
        for layer, (level, ci, co, cup, relu) in enumerate(U.LAYERS):
            o += 27 * ci * co + co
            if level == 0 and layer < 14:
                want = torch.from_numpy(net.gradient(layer, 0, co, level)).cuda().double().sum(0).cpu().numpy()
                err.append(np.linalg.norm(grads[o - co:o] - want) / np.linalg.norm(want))
    assert np.sqrt(np.mean(np.square(err))) <= 3e-7
