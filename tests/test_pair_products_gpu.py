"""Grouped products on pairs of SMs (experts_sm100_pair.cu, experts_sm100_wgrad.cu) at the edges of their tiles: token tiles
of 32 to 256 columns, feature tiles of 128 / 256 with a tail, reductions that end inside a 64-wide block."""
import numpy as np
import pytest
import torch

from helpers import assert_close_bf16, make_layer
from test_parity_gpu import check_routing, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,d,dff,E,k", [
    (1030, 264, 776, 2, 2),    # five equal token tiles per expert; tails in both feature counts
    (769, 1032, 136, 4, 2),    # one feature tile and a bit, K just past a multiple of 64
    (2100, 128, 2056, 24, 5),  # ragged experts
    (300, 1032, 1032, 32, 4),  # no expert above 64 rows: nine narrow stages
    (640, 1032, 1032, 32, 4),  # none above 128: eight
])
def test_forward_at_tile_edges(oracle, T, d, dff, E, k):
    x, w_r, w_g, w_u, w_d, _ = make_layer(T, d, dff, E, k, seed=T)
    rb = oracle.bf16_round
    xb, w_rb = rb(x), rb(w_r)
    r = oracle.moe_forward(xb, w_rb, w_g, w_u, w_d, k, bf16=True)
    y, routing, logits, _ = run_gpu(xb, w_rb, rb(w_g), rb(w_u), rb(w_d), None, k, torch.bfloat16, torch.bfloat16)
    check_routing(routing, logits, r)
    assert_close_bf16(y, r.y)


@pytest.mark.parametrize("T", [1, 31, 32, 33, 64, 65, 100, 128, 129, 255, 256, 257, 481])
def test_training_step_at_tile_edges(oracle, T):
    """Both experts hold all T rows (top-2 of 2), so T is the width that the token tiles are cut from and the length the
    weight gradients reduce over."""
    from helpers import assert_close_bf16_grad
    from test_backward_gpu import NAMES, run_layer
    d, dff, E, k = 136, 328, 2, 2
    x, w_r, w_g, w_u, w_d, _ = make_layer(T, d, dff, E, k, seed=T)
    rb = oracle.bf16_round
    x, w_r, w_g, w_u, w_d = rb(x), rb(w_r * 10), rb(w_g * 3), rb(w_u * 3), rb(w_d * 3)
    dy = rb(np.random.default_rng(T).standard_normal((T, d)).astype(np.float32))
    got, routing = run_layer(T, d, dff, E, k, torch.bfloat16, torch.bfloat16, x, w_r, w_g, w_u, w_d, dy)
    r = oracle.moe_forward(x, w_r, w_g, w_u, w_d, k, bf16=True)
    assert np.array_equal(routing[0], r.topk_idx)
    assert_close_bf16_grad(got["y"], r.y)
    ref = oracle.moe_backward(x, w_r, w_g, w_u, w_d, k, dy, bf16=True, out_bf16=True)
    for name in NAMES:
        assert_close_bf16_grad(got[name], getattr(ref, name))
