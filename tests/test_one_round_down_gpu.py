"""Down product of about one row tile per expert: a tile per CTA where that takes one round and pairs of SMs would take two
(launch_experts_bf16), and pairs on the other side of each bound."""
import pytest
import torch

from helpers import assert_close_bf16, make_layer
from test_parity_gpu import check_routing, run_gpu

pytestmark = pytest.mark.gpu


# 512 rows of top-2 on 8 experts are 15 row tiles at most: too many for a split K from 10 feature tiles on.  88 and 144 tiles run in
# one round; 1026 rows are above one tile per expert, 152 tiles above the SMs.  The 300-row calls split K (one round or not).
@pytest.mark.parametrize("T,d,E", [(512, 2816, 8), (512, 4608, 8), (513, 2816, 8), (512, 4864, 8),
                                   (300, 2560, 8), (513, 2560, 8), (300, 2304, 8), (300, 4864, 8)])
def test_down_product_on_both_sides_of_the_rule(oracle, T, d, E):
    dff, k = 1408, 2
    x, w_r, w_g, w_u, w_d, _ = make_layer(T, d, dff, E, k, seed=T + d)
    rb = oracle.bf16_round
    xb, w_rb = rb(x), rb(w_r)
    r = oracle.moe_forward(xb, w_rb, w_g, w_u, w_d, k, bf16=True)
    y, routing, logits, _ = run_gpu(xb, w_rb, rb(w_g), rb(w_u), rb(w_d), None, k, torch.bfloat16, torch.bfloat16)
    check_routing(routing, logits, r)
    assert_close_bf16(y, r.y)
