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
])
def test_forward_at_tile_edges(oracle, T, d, dff, E, k):
    x, w_r, w_g, w_u, w_d, _ = make_layer(T, d, dff, E, k, seed=T)
    rb = oracle.bf16_round
    xb, w_rb = rb(x), rb(w_r)
    r = oracle.moe_forward(xb, w_rb, w_g, w_u, w_d, k, bf16=True)
    y, routing, logits, _ = run_gpu(xb, w_rb, rb(w_g), rb(w_u), rb(w_d), None, k, torch.bfloat16, torch.bfloat16)
    check_routing(routing, logits, r)
    assert_close_bf16(y, r.y)
