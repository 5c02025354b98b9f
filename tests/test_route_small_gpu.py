"""One-launch routing of a decode step (route_small.cu): rows that end inside a 256-column piece, rows longer than the
shared-memory chunk, expert counts that are no multiple of a warp's, and both sides of the rule for a single block."""
import pytest
import torch

from helpers import assert_close_bf16, make_layer
from test_parity_gpu import check_routing, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("io", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,d,E,k", [
    (1, 72, 1, 1), (8, 264, 128, 16), (3, 4096, 5, 2), (8, 4104, 33, 4), (5, 8200, 65, 3),
    (1, 1536, 8, 2), (1, 1544, 8, 2), (2, 1536, 8, 3), (1, 768, 16, 4), (1, 776, 16, 4), (1, 1000, 5, 2), (1, 128, 17, 3),  # one block, or just not
])
def test_routing_of_a_few_tokens(oracle, T, d, E, k, io):
    dff = 64
    x, w_r, w_g, w_u, w_d, _ = make_layer(T, d, dff, E, k, seed=d + E)
    rb = oracle.bf16_round
    xb, w_rb = rb(x), rb(w_r)
    r = oracle.moe_forward(xb, w_rb, w_g, w_u, w_d, k, bf16=True, out_bf16=io == torch.bfloat16)
    y, routing, logits, n = run_gpu(xb, w_rb, rb(w_g), rb(w_u), rb(w_d), None, k, torch.bfloat16, io)
    check_routing(routing, logits, r)
    assert_close_bf16(y, r.y)
