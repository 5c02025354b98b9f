"""Host-buffer forwards that run in several pieces (forward_host_enqueue in api.cu): every row keeps its bits, and the read-outs
describe what the header says, the whole batch below 8192 tokens and the last chunk from there on."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def make(T, d, dff, E, k, seed=None, t_max=None):
    from omega_ai_b200 import MoELayer
    g = torch.Generator(device="cuda").manual_seed(T if seed is None else seed)
    mk = lambda *s, std=0.02: (torch.randn(*s, device="cuda", generator=g) * std).to(torch.bfloat16)
    weights = lambda: (mk(E, d), mk(E, dff, d), mk(E, dff, d), mk(E, d, dff))
    layer = MoELayer(d, dff, E, k, t_max=t_max or T, compute_dtype=torch.bfloat16)
    layer.setWeights(*weights())
    xd = mk(T, d, std=1.0)
    xh = xd.cpu().pin_memory()
    return layer, weights, xd, xh, torch.empty_like(xh).pin_memory()


def read_logits(layer, T):
    """The logits in a buffer of T rows that are NaN where nothing was written."""
    out = np.full((T, layer.numExperts), np.nan, np.float32)
    assert layer._lib.omoe_get_logits(layer._h, out.ctypes.data_as(C.c_void_p)) == 0
    return out


@pytest.mark.parametrize("T,d,dff,E,k", [
    (4099, 1024, 2816, 8, 2),   # the second chunk is a token shorter
    (6001, 2048, 1408, 4, 1),
    (8191, 1024, 1408, 8, 4),   # the most that is described as a whole
])
def test_small_chunks_match_the_device_forward(T, d, dff, E, k):
    layer, weights, xd, xh, yh = make(T, d, dff, E, k)
    yd = layer.forward_device(xd).clone()
    in_one = layer.launch_count()
    routing, logits = layer.routing(T), layer.logits(T)
    layer.forward_host(xh, yh)
    assert layer.launch_count() >= 2 * in_one - 1, "the batch was not cut"
    assert torch.equal(yd.cpu(), yh)
    for got, want in zip(layer.routing(T), routing):
        assert np.array_equal(got, want)
    assert np.array_equal(layer.logits(T), logits)
    layer.setWeights(*weights())
    assert np.array_equal(layer.logits(T), logits)  # of the weights that the forward had
    for got, want in zip(layer.routing(T), routing):
        assert np.array_equal(got, want)
    n = C.c_void_p()
    assert layer._lib.omoe_get_routing(layer._h, n, n, n, n, n) == 0
    layer.close()


@pytest.mark.parametrize("T", [8192, 9001])
def test_read_outs_of_a_large_batch_describe_its_last_chunk(T):
    """Two chunks of at least 4096 tokens, whatever else they are cut into: a caller's buffers hold one of them."""
    layer, _, xd, xh, yh = make(T, 2048, 1408, 8, 2)
    n = T - (T + 1) // 2
    layer.forward_device(xd[T - n:].contiguous())
    routing, logits, in_one = layer.routing(n), layer.logits(n), layer.launch_count()
    layer.forward_host(xh, yh)
    assert layer.launch_count() > in_one, "the chunk was not cut further"
    got = read_logits(layer, T)
    assert np.array_equal(got[:n], logits) and np.isnan(got[n:]).all()
    for got, want in zip(layer.routing(n), routing):
        assert np.array_equal(got, want)
    assert torch.equal(layer.forward_device(xd).cpu(), yh)
    layer.close()


def test_aux_loss_of_a_cut_batch():
    layer, _, xd, xh, yh = make(4096, 1024, 2816, 8, 2)
    layer.set_training(True)
    layer.set_training(False)
    layer.forward_device(xd)
    want, in_one = layer.aux_loss(), layer.launch_count()
    layer.forward_host(xh, yh)
    assert layer.launch_count() > in_one
    assert layer.aux_loss() == want
    layer.close()


@pytest.mark.parametrize("T", [4096, 8192])
def test_training_forward_is_followed_by_its_backward(T):
    """A training forward runs in the chunks that the header states and no smaller ones; a read-out between it and the backward
    of the rows it kept changes nothing."""
    layer, _, xd, xh, yh = make(T, 2048, 1408, 8, 2)
    last = xd[T - 4096:].contiguous()
    layer.forward_device(last)
    in_one = layer.launch_count()
    layer.forward_host(xh, yh)
    assert layer.launch_count() > in_one, "not cut further when it does not train"
    layer.set_training(True)
    dy = torch.randn_like(last)
    layer.forward_host(xh, yh)
    read_logits(layer, T)
    layer.routing(T)
    dx = layer.backward(last, dy).clone()
    grads = layer.weight_grads()
    layer.forward_device(last)
    assert torch.equal(layer.backward(last, dy), dx)
    for name, g in layer.weight_grads().items():
        assert torch.equal(g, grads[name]), name
    layer.close()


def test_pageable_buffers_and_a_given_minimum_are_not_cut(monkeypatch):
    """Copies from pageable memory hold the host up, so nothing would overlap; OMOE_HOST_CHUNK_MIN is the whole rule when given."""
    T, shape = 4096, (1024, 2816, 8, 2)
    layer, _, xd, xh, yh = make(T, *shape)
    y = layer.forward_device(xd).cpu()
    in_one = layer.launch_count()
    for x, out in ((xh.clone(), yh), (xh, torch.empty_like(y)), (xh.clone(), torch.empty_like(y))):
        layer.forward_host(x, out)
        assert layer.launch_count() == in_one and torch.equal(out, y)
    layer.close()
    monkeypatch.setenv("OMOE_HOST_CHUNK_MIN", "2049")
    layer, _, xd, xh, yh = make(T, *shape)
    layer.forward_host(xh, yh)
    assert layer.launch_count() == in_one and torch.equal(yh, y)
    layer.close()
