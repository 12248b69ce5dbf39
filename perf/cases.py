"""The work a user of this package has it do, as measurable cases.

Four kinds, each through the public entry point a training or serving program calls:

  step    ``FusedFFIShard.step``: one training step of the output layer (forward, loss, both gradients, SR-SGD) from
          a batch of features and COO targets
  layer   ``GroupFixedFanIn`` under autograd with ``SRSgd``: forward, backward, optimizer step
  topk    ``ffi_topk``: the best k labels of every row, without a [B, L] matrix
  rewire  ``GroupFixedFanIn.rewire``: prune, regrow, re-initialise, regroup

The sizes are those of ``haste_b200.synth.WORKLOADS`` and of the tests (31 thousand to 2.8 million labels, fan-in 32 to
128, label groups of 32 to 128, batches of 1 to 1024 rows).  Features are Gaussian, L2-normalised per row or rectified;
weights are uniform in +-1/sqrt(fan_in); index rows are distinct and sorted; label frequencies follow a Zipf law.
"""
import math

import torch

from haste_b200.fused import FusedFFIShard
from haste_b200.infer import ffi_topk
from haste_b200.shared_ffi.optim_sr import SRSgd
from haste_b200.shared_ffi.rewire import GroupFixedFanIn

LR, WD = 0.05, 1e-4


def _step(name, B, D, L, F, G, avg_pos, zipf, x, loss, momentum=0.0, rng="packed"):
    c = dict(kind="step", B=B, D=D, L=L, F=F, G=G, avg_pos=avg_pos, zipf=zipf, x=x, loss=loss, momentum=momentum, rng=rng)
    return dict(c, name=name) if name else c


def _layer(name, B, D, L, F, G, x, x_dtype="bf16"):
    c = dict(kind="layer", B=B, D=D, L=L, F=F, G=G, x=x, x_dtype=x_dtype)
    return dict(c, name=name) if name else c


def _topk(name, B, D, L, F, G, k, x):
    c = dict(kind="topk", B=B, D=D, L=L, F=F, G=G, k=k, x=x)
    return dict(c, name=name) if name else c


def _rewire(name, D, L, F, G, fraction):
    c = dict(kind="rewire", D=D, L=L, F=F, G=G, fraction=fraction)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user's query against a 131 thousand label catalogue: latency is all that counts
        _topk("serve-131k-b1", 1, 768, 131073, 128, 64, 5, "l2norm"),
        # evaluation over a test set: full batches, the 100 best of 670 thousand labels
        _topk("topk-670k-b512", 512, 768, 670091, 64, 128, 100, "l2norm"),
        # training on a small label set with small batches (the configuration that also runs on a CPU)
        _step("step-31k-b64", 64, 768, 30938, 32, 32, 19.0, 1.1, "normal", "bce"),
        # training on 131 thousand labels, wide fan-in
        _step("step-131k-b512", 512, 768, 131073, 128, 64, 5.4, 1.1, "l2norm", "bce"),
        # the headline configuration
        _step("step-670k-b512", 512, 768, 670091, 64, 128, 5.5, 1.0, "l2norm", "squared_hinge"),
        # the layer behind a wide penultimate ReLU layer
        _step("step-500k-b256", 256, 4096, 501070, 128, 64, 4.8, 1.1, "relu", "bce"),
        # the largest label set, the largest batch
        _step("step-2m8-b1024", 1024, 768, 2812281, 64, 128, 36.0, 1.2, "l2norm", "bce"),
        # the last, odd-sized batch of an epoch, trained with momentum
        _step("step-131k-b333-mom", 333, 768, 131073, 64, 128, 5.4, 1.1, "l2norm", "squared_hinge", momentum=0.9),
        # the layer inside a user's own model and training loop: fp32 activations, a small label set
        _layer("layer-31k-b64", 64, 768, 30938, 32, 32, "normal", "fp32"),
        # the same at the layer class's default group size
        _layer("layer-131k-b256", 256, 768, 131073, 64, 32, "l2norm"),
        # the same at the headline size: [B, L] logits and gradients of 686 MB each
        _layer("layer-670k-b512", 512, 768, 670091, 64, 128, "l2norm"),
        # the rewiring of a 500 thousand label layer, every thousand steps
        _rewire("rewire-500k", 4096, 501070, 128, 64, 0.15),
    ]


# (group size, fan-in) pairs of the workloads and of the layer's default group size
_SHAPES = [(128, 64), (64, 128), (32, 32), (32, 64), (64, 64), (32, 128)]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _width(rng):
    """Feature width: mostly that of an encoder or a penultimate layer, now and then anything."""
    return rng.choice([512, 768, 1024, 2048, 4096]) if rng.random() < 0.75 else rng.randrange(256, 4097)


def _batch(rng, lo, hi):
    """Mostly full batches (multiples of 8), else what is left at the end of an epoch."""
    b = _log_int(rng, lo, hi)
    return max(8, b // 8 * 8) if rng.random() < 0.6 and b >= 8 else b


def draw(rng):
    kind = rng.choices(["step", "layer", "topk", "rewire"], [5, 3, 2, 1])[0]
    G, F = rng.choice(_SHAPES)
    D = _width(rng)
    x = rng.choice(["normal", "l2norm", "relu"])
    if kind == "step":
        B = _batch(rng, 32, 1024)
        L = _log_int(rng, 4096, int(min(2.8e6, 5e8 / B)))
        return _step(None, B, D, L, F, G, round(rng.uniform(2.0, 36.0), 1), round(rng.uniform(1.0, 1.2), 2), x,
                     rng.choice(["bce", "squared_hinge"]), momentum=rng.choice([0.0, 0.0, 0.9]), rng=rng.choice(["packed", "packed", "reference"]))
    if kind == "layer":
        B = _batch(rng, 32, 1024)
        return _layer(None, B, D, _log_int(rng, 4096, int(min(6.7e5, 1e8 / B))), F, G, x, rng.choice(["bf16", "bf16", "fp32"]))
    if kind == "topk":
        B = _batch(rng, 1, 1024)
        return _topk(None, B, D, _log_int(rng, 4096, int(min(2.8e6, 3e8 / B))), F, G, rng.choice([1, 5, 10, 50, 100]), x)
    return _rewire(None, D, _log_int(rng, 4096, 670000), F, G, round(rng.uniform(0.05, 0.3), 2))


def _features(B, D, kind, gen):
    X = torch.randn(B, D, generator=gen, device="cuda")
    if kind == "l2norm":
        X = X / X.norm(dim=1, keepdim=True)
    elif kind == "relu":
        X = X.clamp_(min=0)
    return X


def _parameters(c, gen):
    """(index table int32 [NG, F], weights bf16 [L, F], bias bf16 [L])"""
    L, F, D = c["L"], c["F"], c["D"]
    NG = (L + c["G"] - 1) // c["G"]
    loc = torch.empty(NG, F, dtype=torch.int32, device="cuda")
    for g in range(0, NG, 16384):
        n = min(16384, NG - g)
        loc[g:g + n] = torch.rand(n, D, generator=gen, device="cuda").topk(F, dim=1).indices.sort(dim=1).values.to(torch.int32)
    W = ((torch.rand(L, F, generator=gen, device="cuda") * 2 - 1) / math.sqrt(F)).to(torch.bfloat16)
    bias = (torch.randn(L, generator=gen, device="cuda") * 0.01).to(torch.bfloat16)
    return loc, W, bias


def _targets(c, gen):
    """int32 [nnz, 2] of (row, label): Poisson many positives per row, Zipf label frequencies, no pair twice."""
    B, L = c["B"], c["L"]
    cdf = torch.cumsum(torch.arange(1, L + 1, device="cuda", dtype=torch.float64).pow(-c["zipf"]), 0)
    n = torch.poisson(torch.full((B,), float(c["avg_pos"]), device="cuda"), generator=gen).clamp_(min=1).long()
    rows = torch.repeat_interleave(torch.arange(B, device="cuda"), n)
    u = torch.rand(rows.numel(), generator=gen, device="cuda", dtype=torch.float64) * cdf[-1]
    cols = torch.searchsorted(cdf, u).clamp_(max=L - 1)
    key = torch.unique(rows * L + cols)
    return torch.stack([key // L, key % L], 1).to(torch.int32)


def _module(c, loc, W, bias, **kwargs):
    m = GroupFixedFanIn(c["D"], c["L"], c["F"], device="cuda", dtype=torch.bfloat16, group_size=c["G"], prune_mode="fraction", **kwargs)
    with torch.no_grad():
        m.weights.copy_(W)
        m.bias.copy_(bias)
        m.group_locations.copy_(loc)
    return m


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    loc, W, bias = _parameters(c, gen)
    if c["kind"] == "rewire":
        return dict(case=c, layer=_module(c, loc, W, bias, rewire_fraction=c["fraction"], init_mode="zero", regrow="unused", regroup=True, seed=int(seed)))
    X = _features(c["B"], c["D"], c["x"], gen)
    if c["kind"] == "topk":
        return dict(case=c, x=X.to(torch.bfloat16), loc=loc, w=W, bias=bias)
    if c["kind"] == "step":
        # squared hinge is averaged over the [B, L] matrix, BCE over the batch rows
        scale = 1.0 / (c["B"] * c["L"]) if c["loss"] == "squared_hinge" else 1.0 / c["B"]
        shard = FusedFFIShard(loc, W, bias, c["G"], c["D"], loss=c["loss"], lr=LR, weight_decay=WD, momentum=c["momentum"], seed=123,
                              rng=c["rng"], grad_scale=scale)
        return dict(case=c, shard=shard, x=X.to(torch.bfloat16), targets=_targets(c, gen))
    layer = _module(c, loc, W, bias, rewire_fraction=0.15)
    dy = torch.empty(c["B"], c["L"], dtype=torch.bfloat16, device="cuda").normal_(0.0, 1e-3, generator=gen)
    x = X if c["x_dtype"] == "fp32" else X.to(torch.bfloat16)
    return dict(case=c, layer=layer, opt=SRSgd(layer.parameters(), lr=LR, weight_decay=WD), x=x.requires_grad_(True), dy=dy)


def run(state):
    kind = state["case"]["kind"]
    if kind == "step":
        sh = state["shard"]
        dxt, loss = sh.step(state["x"], state["targets"])
        out = dict(dxt=dxt, loss=loss, w=sh.w, bias=sh.bias)
        if sh.mom_w is not None:
            out.update(mom_w=sh.mom_w, mom_b=sh.mom_b)
        return out
    if kind == "layer":
        layer, x = state["layer"], state["x"]
        x.grad = None
        state["opt"].zero_grad()
        z = layer(x)
        z.backward(state["dy"])
        state["opt"].step()
        return dict(z=z.detach(), dx=x.grad, w=layer.weights.data, bias=layer.bias.data)
    if kind == "topk":
        values, labels = ffi_topk(state["loc"], state["w"], state["bias"], state["x"], state["case"]["k"], state["case"]["G"])
        return dict(values=values, labels=labels)
    changed = state["layer"].rewire()
    return dict(w=state["layer"].weights.data, loc=state["layer"].group_locations, changed=changed)


def work(case):
    c = case
    L, F, G, D = c["L"], c["F"], c["G"], c["D"]
    NG = (L + G - 1) // G
    w, loc, bias = 2 * L * F, 4 * NG * F, 2 * L
    if c["kind"] == "rewire":
        return dict(bytes=2 * w + 2 * loc, flops=0)
    B = c["B"]
    if c["kind"] == "topk":
        return dict(bytes=w + loc + bias + 2 * B * D + 8 * B * c["k"], flops=2 * B * L * F)
    if c["kind"] == "step":
        mom = 8 * (L * F + L) if c["momentum"] else 0
        return dict(bytes=2 * w + loc + 2 * bias + mom + 2 * B * D + 4 * B * D + 8 * int(B * c["avg_pos"]), flops=6 * B * L * F)
    # logits out, their gradient in; weights read by the forward and by the backward, then updated from their gradient
    x = (4 if c["x_dtype"] == "fp32" else 2) * B * D
    return dict(bytes=2 * 2 * B * L + 5 * w + 2 * loc + 4 * bias + 2 * x, flops=6 * B * L * F)


def tolerance(case):
    """Against the same path in 64 bits (no rounding of logits, loss gradients or weights), on the listed sizes: rel up to
    2.4e-3 and max up to 8.8e-3 of a step or layer (one bf16 rounding is up to 2^-8 of a value, a stochastic one 2^-7);
    top-k values and labels identical, and a sum in another order may turn a logit into its bf16 neighbour."""
    if case["kind"] == "rewire":
        return "exact"
    if case["kind"] == "topk":
        return {"rel": 1e-3, "max": 1e-2, "differ": 2e-3}
    return {"rel": 1e-2, "max": 4e-2}
