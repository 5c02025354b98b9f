"""Row tiles of the fp32 products (experts_f32.cu): how a block finds its expert, and layers whose t_max is far above a call's rows."""
import numpy as np
import pytest
import torch

from helpers import assert_close_f32, make_layer
from test_backward_gpu import NAMES, close_scaled, run_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,d,dff,E,k", [
    (1, 8, 8, 128, 3),      # three rows over four groups of 32 experts
    (33, 72, 136, 2, 2),    # every expert holds 33 rows: a tile of 32 and one row
    (64, 64, 64, 40, 7),    # experts past the first 32
    (700, 128, 72, 4, 1),   # several tiles per expert, one column tile and a bit
])
def test_row_tiles_find_their_experts(oracle, T, d, dff, E, k):
    x, w_r, w_g, w_u, w_d, bias = make_layer(T, d, dff, E, k, seed=T, zipf=True)
    w_r, w_g, w_u, w_d = ((w * s).astype(np.float32) for w, s in ((w_r, 10), (w_g, 3), (w_u, 3), (w_d, 3)))
    dy = np.random.default_rng(T).standard_normal((T, d)).astype(np.float32)
    f32 = torch.float32
    got, routing = run_layer(T, d, dff, E, k, f32, f32, x, w_r, w_g, w_u, w_d, dy, bias)
    r = oracle.moe_forward(x, w_r, w_g, w_u, w_d, k, bias=bias)
    assert np.array_equal(routing[0], r.topk_idx)
    assert_close_f32(got["y"], r.y)
    ref = oracle.moe_backward(x, w_r, w_g, w_u, w_d, k, dy, bias=bias)
    for name in NAMES:
        close_scaled(got[name], getattr(ref, name), name, 2e-4)


def test_layer_of_two_million_rows(oracle):
    """The buffers hold 2.1 million rows, 65,628 tiles of 32: more than a grid's second dimension takes."""
    from omega_ai_b200 import MoELayer
    T, d, dff, E, k = 5, 8, 8, 4, 2
    x, w_r, w_g, w_u, w_d, _ = make_layer(T, d, dff, E, k, seed=7)
    dev = lambda a: torch.from_numpy(a).cuda()
    layer = MoELayer(d, dff, E, k, t_max=1_050_000, compute_dtype=torch.float32)
    layer.setWeights(dev(w_r), dev(w_g), dev(w_u), dev(w_d))
    y = layer.forward_device(dev(x))
    assert_close_f32(y.cpu().numpy(), oracle.moe_forward(x, w_r, w_g, w_u, w_d, k).y)
    layer.set_training(True)
    assert torch.equal(layer.forward_device(dev(x)), y)
    dx = layer.backward(dev(x), dev(x))
    close_scaled(dx.cpu().numpy(), oracle.moe_backward(x, w_r, w_g, w_u, w_d, k, x).dx, "dx", 2e-4)
    layer.close()
