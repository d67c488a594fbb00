"""The network's tensor-core kernels (forward, input gradient, weight and bias gradient) against a float64 convolution of
the same inputs on the GPU, at the level widths 128 to 8 and every pair of channel counts that the network has: one input or
two, upsampled or not, one slice of input channels or twelve, items that end inside the volume and at its faces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ACT_C = [16, 16, 16, 16, 32, 32, 32, 64, 64, 64, 128, 128, 64, 64, 32, 32, 16, 16]
ACT_L = [0, 0, 0, 1, 1, 1, 2, 2, 2, 3, 3, 3, 2, 2, 1, 1, 0, 0]
IN1 = [0, 1, 3, 4, 6, 7, 9, 10, 11, 12, 13, 14, 15, 16, 17]
IN2 = [None] * 8 + [8, None, 5, None, 2, None, None]
OUT = [1, 2, 4, 5, 7, 8, 10, 11, 12, 13, 14, 15, 16, 17, None]


def windows(x):
    import torch
    e = x.shape[0]
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    for t in range(27):
        yield xp[t // 9:t // 9 + e, t // 3 % 3:t // 3 % 3 + e, t % 3:t % 3 + e]


@pytest.mark.parametrize("edge", [64, 128])
def test_kernels_match_float64(edge):
    """Tolerances (relative L2), as for the kernels at edge 32: BF16 outputs 2e-3 (half a unit in the last place of eight
    bits, uniformly spread, is 1.7e-3), FP32 output 1e-5, weight and bias gradients 1e-4 (FP32 accumulation)."""
    import torch
    from oracle import unet_ref as U
    from vortegrid_gb300 import warmstart as ws
    net, grid = ws.Network(edge), ws.field_grid(edge + 1)
    params = ws.init_params(seed=11, zero_output=False)
    rng = np.random.default_rng(5)
    o = 0
    for ci, co in ws.LAYERS:
        o += 27 * co * ci
        params[o:o + co] = rng.normal(0, 0.05, co)
        o += co
    net.set_params(params, 0.5)
    n3 = (edge + 1) ** 3
    rhs = torch.from_numpy(rng.normal(0, 1, (n3, 3)).astype(np.float32)).cuda()
    vp = torch.from_numpy(rng.normal(0, 1e-3, (n3, 3)).astype(np.float32)).cuda()
    net.backward(grid, rhs, vp, want_loss=True)
    acts = [torch.from_numpy(net.activation(k, ACT_C[k], ACT_L[k])).cuda().double() for k in range(18)]
    grads = net.grads()
    rel = lambda a, b: float((a - b).norm() / b.norm())  # noqa: E731
    bad, o = {}, 0

    def check(name, err, bound):
        if not err < bound:
            bad[name] = (err, bound)
    for l, (level, ci, co, cup, relu) in enumerate(U.LAYERS):
        e = edge >> level
        nw = 27 * ci * co
        w = torch.from_numpy(params[o:o + nw].reshape(27, co, ci)).cuda().bfloat16().double()
        b = torch.from_numpy(params[o + nw:o + nw + co]).cuda().double()
        gw = torch.from_numpy(grads[o:o + nw].reshape(27, co, ci)).cuda().double()
        gb = torch.from_numpy(grads[o + nw:o + nw + co]).cuda().double()
        o += nw + co
        x = acts[IN1[l]]
        if cup:
            x = x.reshape(e // 2, e // 2, e // 2, -1)
            x = x.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)
            x = torch.cat([x, acts[IN2[l]].reshape(e, e, e, -1)], 3)
        x = x.reshape(e, e, e, ci)
        g = torch.from_numpy(net.gradient(l, 0, co, level)).cuda().double()
        y = b.expand(e, e, e, co).clone()
        dw = []
        for t, win in enumerate(windows(x)):
            y += win @ w[t].T
            dw.append(g.T @ win.reshape(-1, ci))
        if relu:
            y = torch.nn.functional.leaky_relu(y, U.SLOPE)
        got = acts[OUT[l]] if OUT[l] is not None else torch.from_numpy(net.output()).cuda().double()
        check(f"forward {l}", rel(got.reshape(e, e, e, co), y), 2e-3 if OUT[l] is not None else 1e-5)
        check(f"weight gradient {l}", rel(gw, torch.stack(dw)), 1e-4)
        check(f"bias gradient {l}", rel(gb, g.sum(0)), 1e-4)
        if l == 0:
            continue
        dx = torch.zeros((e, e, e, ci), dtype=torch.float64, device="cuda")
        for t, win in enumerate(windows(g.reshape(e, e, e, co))):
            dx += win @ w[26 - t]
        if cup or l in (2, 4, 6):
            got = net.gradient(l, 1, ci, level)
        else:
            got = net.gradient(l - 1, 0, ci, level)
            dx = torch.where(acts[IN1[l]].reshape(e, e, e, ci) > 0, dx, U.SLOPE * dx)
        check(f"input gradient {l}", rel(torch.from_numpy(got).cuda().double().reshape(e, e, e, ci), dx), 2e-3)
    assert not bad, bad


@pytest.mark.parametrize("scale", [1e-25, 1.0, 1e25])
def test_guess_scales_with_the_right_hand_side(scale):
    """The guess is linear in the field's magnitude, also where the squares of its values leave the range of floats."""
    import torch
    from vortegrid_gb300 import warmstart as ws
    net, grid = ws.Network(32), ws.field_grid(33)
    net.set_params(ws.init_params(seed=3, zero_output=False), 0.5)
    rng = np.random.default_rng(8)
    rhs = torch.from_numpy(rng.normal(0, 1, (33 ** 3, 3)).astype(np.float32)).cuda()
    want, got = torch.zeros_like(rhs), torch.zeros_like(rhs)
    net.guess(grid, rhs, want)
    net.guess(grid, rhs * scale, got)
    net.synchronize()
    # the scaled inputs may round to a neighbouring BF16 value (2^-9 of a value), a few percent of them
    assert float((got.double() / scale - want.double()).norm() / want.double().norm()) < 5e-3
