"""Host-buffer forwards cut into chunks below the general minimum (chunk_pays in api.cu): every row keeps its bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,d,dff,E,k", [(4099, 1024, 128, 8, 2), (6001, 2048, 64, 4, 1), (4095, 1024, 128, 8, 2)])
def test_small_chunks_match_the_device_forward(T, d, dff, E, k):
    from omega_ai_b200 import MoELayer
    g = torch.Generator(device="cuda").manual_seed(T)
    mk = lambda *s: (torch.randn(*s, device="cuda", generator=g) * 0.02).to(torch.bfloat16)
    layer = MoELayer(d, dff, E, k, t_max=T, compute_dtype=torch.bfloat16)
    layer.setWeights(mk(E, d), mk(E, dff, d), mk(E, dff, d), mk(E, d, dff))
    xd = torch.randn(T, d, device="cuda", generator=g).to(torch.bfloat16)
    yd = layer.forward_device(xd).clone()
    routing, logits = layer.routing(T), layer.logits(T)
    xh = xd.cpu().pin_memory()
    yh = torch.empty_like(xh).pin_memory()
    layer.forward_host(xh, yh)
    assert torch.equal(yd.cpu(), yh)
    for got, want in zip(layer.routing(T), routing):  # of the whole batch, not of the last chunk
        assert np.array_equal(got, want)
    layer.forward_host(xh, yh)
    layer.setWeights(mk(E, d), mk(E, dff, d), mk(E, dff, d), mk(E, d, dff))
    assert np.array_equal(layer.logits(T), logits)  # of the weights that the forward had
    layer.close()


def test_training_forward_is_not_cut():
    """The backward follows a forward of the whole batch, host buffers or not."""
    from omega_ai_b200 import MoELayer
    T, d, dff, E, k = 4096, 1024, 128, 8, 2
    g = torch.Generator(device="cuda").manual_seed(1)
    mk = lambda *s: (torch.randn(*s, device="cuda", generator=g) * 0.02).to(torch.bfloat16)
    layer = MoELayer(d, dff, E, k, t_max=T, compute_dtype=torch.bfloat16)
    layer.setWeights(mk(E, d), mk(E, dff, d), mk(E, dff, d), mk(E, d, dff))
    layer.set_training(True)
    xd, dy = mk(T, d), mk(T, d)
    xh = xd.cpu().pin_memory()
    layer.forward_host(xh, torch.empty_like(xh).pin_memory())
    dx = layer.backward(xd, dy).clone()
    layer.forward_device(xd)
    assert torch.equal(layer.backward(xd, dy), dx)
    layer.close()
