"""What the layer's speed is judged on: calls a program makes through the package's entry points, over the sizes it makes
them at.

A case is a dict of plain values:

  path     forward | block | train | train_block | host    (see run())
  compute  "bf16" or "f32": arithmetic of the layer;  io: element type of the rows handed over
  T, d, dff, E, k                                          tokens, widths, experts, picks per token
  zipf     the router's bias skews the load of the experts (2 * rank^-1.1);  renorm: gate weights sum to 1
  aux      weight of the load-balancing loss in the objective (training only)

Inputs and weights follow the distributions of the benchmark's workloads: x ~ N(0, 1), weights ~ N(0, 0.02).
"""
import math

import torch

from omega_ai_b200 import MoELayer, Tensor

DTYPE = {"bf16": torch.bfloat16, "f32": torch.float32}


def _case(name, path, T, d, dff, E, k, compute="bf16", io=None, zipf=False, renorm=True, aux=0.0):
    c = dict(path=path, T=T, d=d, dff=dff, E=E, k=k, compute=compute, io=io or compute, zipf=zipf, renorm=renorm, aux=aux)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small layer in the engine's own precision, driven through Layer.forward(Tensor): launches and latency
        _case("f32_forward_64", "forward", 64, 128, 256, 8, 2, compute="f32"),
        # one request generating: one token per step through a Mixtral-shaped layer
        _case("decode_1", "forward", 1, 4096, 14336, 8, 2),
        # a serving batch of 64 sequences, one token each
        _case("decode_64", "forward", 64, 4096, 14336, 8, 2),
        # a few sequences on a layer of many small experts
        _case("decode_fine_8", "forward", 8, 2048, 1408, 64, 6, zipf=True),
        # prompt or evaluation pass, batch 8 x 512 tokens, mid-size layer
        _case("forward_mid_4096", "forward", 4096, 1024, 2816, 8, 2),
        # the same on many small experts with a skewed load
        _case("forward_fine_8192", "forward", 8192, 2048, 1408, 64, 6, zipf=True),
        # the largest inference pass: the benchmark's default workload
        _case("forward_large_16384", "forward", 16384, 4096, 14336, 8, 2),
        # feed-forward half of a transformer block on fp32 Tensors (the engine's only row type), sizes off every tile,
        # gate weights not renormalised
        _case("block_ragged_1531", "block", 1531, 1544, 4104, 12, 3, io="f32", zipf=True, renorm=False),
        # a training step of the mid-size layer: forward, backward, all gradients
        _case("train_mid_4096", "train", 4096, 1024, 2816, 8, 2, aux=0.01),
        # a training step of the Mixtral-shaped layer
        _case("train_large_8192", "train", 8192, 4096, 14336, 8, 2, aux=0.01),
        # a training step of a small fp32 block
        _case("train_block_f32_300", "train_block", 300, 256, 384, 8, 2, compute="f32"),
        # rows in pinned host memory, in and out, one call at a time
        _case("host_mid_4096", "host", 4096, 1024, 2816, 8, 2),
    ]


# A drawn case stays within the weights and the multiply-adds of the largest listed ones.
_WEIGHTS_MAX = 8 * 4096 * 14336
_FLOPS_MAX = 6.0 * 16384 * 2 * 4096 * 14336


def _log(rng, lo, hi, step=1):
    """Uniform over the logarithm of [lo, hi], a multiple of `step`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, step * round(v / step)))


def draw(rng):
    path = rng.choice(["forward", "forward", "forward", "decode", "decode", "block", "train", "train_block", "host", "f32"])
    if path == "f32":  # layers in the engine's precision are small
        path = rng.choice(["forward", "block", "train", "train_block"])
        d, dff, E = _log(rng, 64, 512, 8), _log(rng, 64, 1024, 8), rng.choice([4, 8, 16])
        return _case(None, path, _log(rng, 8, 1024), d, dff, E, rng.randint(1, min(4, E)), compute="f32",
                     aux=0.01 if path == "train" else 0.0)
    while True:
        d, dff, E = _log(rng, 512, 4096, 8), _log(rng, 704, 14336, 8), rng.choice([8, 8, 16, 32, 64])
        k = rng.randint(1, 2) if E == 8 else rng.choice([2, 4, 6])
        if E * d * dff <= _WEIGHTS_MAX:
            break
    train = path.startswith("train")
    top = _FLOPS_MAX / (3.0 if train else 1.0) / (6.0 * k * d * dff)
    if path == "decode":
        T = _log(rng, 1, 256)
    else:
        T = _log(rng, 257, max(258, int(min(8192 if train or path == "host" else 16384, top))))
    io = "f32" if path in ("block", "train_block") and rng.random() < 0.5 else "bf16"
    return _case(None, "forward" if path == "decode" else path, T, d, dff, E, k, io=io, zipf=E > 8 and rng.random() < 0.5,
                 renorm=rng.random() < 0.8, aux=0.01 if path == "train" else 0.0)


def _inputs(case, seed):
    """Router bias, weights (router, gate, up, down), rows, gradient of the output and the block's gamma; None where the
    path has none."""
    T, d, dff, E = case["T"], case["d"], case["dff"], case["E"]
    dt, io = DTYPE[case["compute"]], DTYPE[case["io"]]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rn(*shape, std=1.0, dtype=io):
        return torch.randn(*shape, generator=g, device="cuda").mul_(std).to(dtype)

    bias = None
    if case["zipf"]:
        rank = torch.randperm(E, generator=g, device="cuda") + 1
        bias = (2.0 * rank.double() ** -1.1).to(dt)
    weights = [rn(E, d, std=0.02, dtype=dt), rn(E, dff, d, std=0.02, dtype=dt), rn(E, dff, d, std=0.02, dtype=dt),
               rn(E, d, dff, std=0.02, dtype=dt)]
    x = rn(T, d)
    dy = rn(T, d) if case["path"].startswith("train") else None
    gamma = 1.0 + rn(d, std=0.1, dtype=torch.float32) if "block" in case["path"] else None
    return bias, weights, x, dy, gamma


def prepare(case, seed):
    """The layer with its weights, and one batch of rows."""
    layer = MoELayer(case["d"], case["dff"], case["E"], case["k"], bias=case["zipf"], t_max=case["T"],
                     compute_dtype=DTYPE[case["compute"]], renormalize=case["renorm"])
    bias, weights, x, dy, gamma = _inputs(case, seed)
    layer.setWeights(*weights, bias)
    s = {"case": case, "layer": layer, "x": x}
    if dy is not None:
        layer.set_training(True)
        layer.set_aux_loss(case["aux"])
        s["dy"] = dy
    if gamma is not None:
        s["gamma"] = gamma
    if case["path"] == "host":
        s["x"] = s["x"].cpu().pin_memory()
        s["y"] = torch.empty_like(s["x"]).pin_memory()
    if case["path"] == "forward" and case["compute"] == "f32":
        s["tensor"] = Tensor.from_device(s["x"])
    return s


def run(s):
    layer, x, path = s["layer"], s["x"], s["case"]["path"]
    if path == "forward":
        if "tensor" in s:  # the engine's operator surface
            return layer.forward(s["tensor"]).view2d()
        return layer.forward_device(x)
    if path == "block":
        return layer.forward_block(x, s["gamma"])
    if path == "host":
        return layer.forward_host(x, s["y"])
    if path == "train":
        y = layer.forward_device(x)
        dx = layer.backward(x, s["dy"])
        return dict(layer.weight_grads(), y=y, dx=dx)
    y = layer.forward_block(x, s["gamma"])
    dx, dgamma = layer.backward_block(x, s["gamma"], s["dy"])
    return dict(layer.weight_grads(), y=y, dx=dx, dgamma=dgamma)


def work(case):
    T, d, dff, E, k = (case[n] for n in ("T", "d", "dff", "E", "k"))
    ws, rs = (2 if case[n] == "bf16" else 4 for n in ("compute", "io"))
    active = E * (1.0 - (1.0 - k / E) ** T)  # experts that some token picked
    per_expert = 3.0 * d * dff
    nbytes = active * per_expert * ws + E * d * 4.0 + 2.0 * T * d * rs
    flops = 6.0 * T * k * d * dff + 2.0 * T * d * E
    if case["path"].startswith("train"):
        nbytes += 2.0 * T * d * rs + 4.0 * (E * per_expert + E * d + E)  # dy in, dx out, fp32 gradients out
        flops *= 3.0
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # Four times what the outputs were measured to be off by from the same layer in 64 bits without the intermediate
    # roundings: f32 4e-7 (largest 2e-6) forward and 6e-7 (4e-6) backward; bf16 3e-3 (1.4e-2) and 4.1e-3 (2.4e-2). The
    # f32 sums get room for the longest reductions drawn.
    if case["compute"] == "f32":
        return {"rel": 5e-6, "max": 4e-5}
    return {"rel": 1.7e-2, "max": 0.1} if case["path"].startswith("train") else {"rel": 1.2e-2, "max": 6e-2}


def exact(case, seed):
    """The same outputs in 64 bits.  Picks are taken from the logits of the rows the router sees, which the block form
    hands over in the layer's element type; nothing else is rounded."""
    T, d, E, k = (case[n] for n in ("T", "d", "E", "k"))
    bias, (w_r, w_g, w_u, w_d), x, dy, gamma = _inputs(case, seed)
    x0 = x.double()
    xn = x0
    if gamma is not None:
        inv = (x0.square().mean(1, keepdim=True) + 1e-5).rsqrt()
        xn = x0 * inv * gamma.double()
    rows = xn.to(w_r.dtype).double() if gamma is not None else xn
    b = bias.double() if bias is not None else 0.0
    picks = (rows @ w_r.double().T + b).topk(k, dim=1).indices
    p = (xn @ w_r.double().T + b).softmax(1)
    pk = p.gather(1, picks)
    w = pk / pk.sum(1, keepdim=True) if case["renorm"] else pk
    y = x0.clone() if gamma is not None else torch.zeros_like(x0)
    if dy is not None:
        g0 = dy.double()
        dw, dx = torch.zeros_like(w), torch.zeros_like(x0)
        keep = torch.float64 if case["compute"] == "f32" else torch.float32  # rounds the large ones once, at the end
        grads = {n: torch.zeros(m.shape, dtype=keep, device="cuda") for n, m in
                 (("d_gate", w_g), ("d_up", w_u), ("d_down", w_d))}
    for e in range(E):
        t, j = (picks == e).nonzero(as_tuple=True)
        if not len(t):
            continue
        wg, wu, wd, xe, we = w_g[e].double(), w_u[e].double(), w_d[e].double(), xn[t], w[t, j].unsqueeze(1)
        g, u = xe @ wg.T, xe @ wu.T
        sg = g.sigmoid()
        h = g * sg * u
        ye = h @ wd.T
        y.index_add_(0, t, we * ye)
        if dy is not None:
            dye = g0[t]
            dw[t, j] = (dye * ye).sum(1)
            dye = we * dye
            dh = dye @ wd
            dg, du = dh * u * sg * (1.0 + g * (1.0 - sg)), dh * g * sg
            grads["d_gate"][e], grads["d_up"][e], grads["d_down"][e] = dg.T @ xe, du.T @ xe, dye.T @ h
            dx.index_add_(0, t, dg @ wg + du @ wu)
    if dy is None:
        return y.cpu() if case["path"] == "host" else y
    dpk = (dw - (dw * w).sum(1, keepdim=True)) / pk.sum(1, keepdim=True) if case["renorm"] else dw
    load = torch.bincount(picks.flatten(), minlength=E).double() / (T * k)
    dp = (case["aux"] * E / T * load).expand(T, E).scatter_add(1, picks, dpk)
    dl = p * (dp - (p * dp).sum(1, keepdim=True))
    grads["d_router"], grads["d_bias"] = dl.T @ xn, dl.sum(0)
    dx += dl @ w_r.double()
    grads = {n: grads[n] for n in ("d_router", "d_bias", "d_gate", "d_up", "d_down")}
    if gamma is None:
        return dict(grads, y=y, dx=dx)
    dgamma = (x0 * inv * dx).sum(0)
    dn = dx * gamma.double()
    dx = g0 + inv * (dn - x0 * inv.square() * (dn * x0).mean(1, keepdim=True))
    return dict(grads, y=y, dx=dx, dgamma=dgamma)
