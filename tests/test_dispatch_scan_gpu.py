"""Dispatch that does the scan's work itself (permute.cu) on both sides of its rule: histograms of up to 2048 counts, router
blocks of 8 tokens or more."""
import pytest
import torch

from helpers import assert_close_f32, make_layer
from test_parity_gpu import check_routing, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,k", [(9, 8, 2), (1024, 16, 4), (1033, 16, 16), (2048, 8, 1), (4200, 8, 3), (40, 33, 2)])
def test_positions_on_both_sides_of_the_rule(oracle, T, E, k):
    d, dff = 64, 64
    x, w_r, w_g, w_u, w_d, bias = make_layer(T, d, dff, E, k, seed=T, zipf=True)
    r = oracle.moe_forward(x, w_r, w_g, w_u, w_d, k, bias=bias)
    y, routing, logits, _ = run_gpu(x, w_r, w_g, w_u, w_d, bias, k, torch.float32, torch.float32)
    check_routing(routing, logits, r)
    assert_close_f32(y, r.y)
