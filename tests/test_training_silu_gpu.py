"""SiLU and its derivative in a bf16 training step, element by element, down to where exp(-g) is near the largest float."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_training_silu_has_fp32_accuracy():
    """One token, one expert: with x = e0, dy = e0 and a first row of W_down of ones the weight gradients are h, dg and du
    themselves.  g runs over the bf16 numbers from -88.5 to 30; u = 2^60 keeps every result a normal number."""
    from omega_ai_b200 import MoELayer
    d, dff = 64, 1024
    g = torch.linspace(-88.5, 30.0, dff).to(torch.bfloat16)
    w_g, w_u, w_d = torch.zeros(1, dff, d), torch.zeros(1, dff, d), torch.zeros(1, d, dff)
    w_g[0, :, 0], w_u[0, :, 0], w_d[0, 0, :] = g.float(), 2.0 ** 60, 1.0
    dev = lambda t: t.to(torch.bfloat16).cuda().contiguous()
    layer = MoELayer(d, dff, 1, 1, t_max=1, compute_dtype=torch.bfloat16)
    layer.setWeights(dev(torch.zeros(1, d)), dev(w_g), dev(w_u), dev(w_d))
    layer.set_training(True)
    e0 = torch.zeros(1, d)
    e0[0, 0] = 1.0
    x = dev(e0)
    layer.forward_device(x)
    layer.backward(x, x)
    got = layer.weight_grads()
    x64, u = g.double().numpy(), 2.0 ** 60
    sg = 1.0 / (1.0 + np.exp(-x64))
    want = {"d_down": (got["d_down"][0, 0, :], x64 * sg * u), "d_up": (got["d_up"][0, :, 0], x64 * sg),
            "d_gate": (got["d_gate"][0, :, 0], u * sg * (1.0 + x64 * (1.0 - sg)))}
    for name, (have, ref) in want.items():
        have = have.double().cpu().numpy()
        # one rounding to bf16 (8 significant bits: half a unit in the last place is up to 2^-8 of the value), and a few to
        # fp32 (16 units of 24 bits) of the terms, which cancel in the derivative near g = -1.28
        terms = np.abs(ref) + (u * sg * (1.0 + np.abs(x64)) if name == "d_gate" else 0.0)
        bound = 2.0 ** -8 * np.abs(ref) + 2.0 ** -20 * terms
        err = np.abs(have - ref)
        assert (err <= bound).all(), f"{name}: {(err / np.abs(ref)).max():.2e} off at g = {x64[np.argmax(err / bound)]}"
    layer.close()
