"""GPU parity tests of the tcgen05 kernels at the layer shapes whose tiles hold 64 labels or two label groups, at batch
sizes that are not multiples of 8 (padded rows of xt), and of the filtered top-k.  Tolerances: bf16 inputs, fp32
accumulation, bf16 logits and loss gradients — rel 1e-2 / abs 1e-3 of the magnitude, as for the other shapes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import ffi_oracle as fo

# (G, F, L): one tile, an odd number of groups (the last tile of a pair holds one), ragged last groups, more tiles than SMs
LAYERS = [(32, 32, 40), (32, 32, 32 * 401 + 7), (32, 64, 32 * 7), (32, 64, 32 * 310 + 1), (64, 64, 64 * 160 + 33), (64, 64, 8),
          (32, 128, 32 * 160 + 9), (32, 128, 17), (128, 64, 128 * 5 + 3), (64, 128, 64 * 9 + 1)]


def _close(got, want, what, rel=1e-2):
    got, want = got.float().cpu(), want.float().cpu()
    bad = (got - want).abs() > 1e-3 * max(1.0, float(want.abs().max())) + rel * want.abs()
    assert not bad.any(), f"{what}: {int(bad.sum())}/{bad.numel()} outside tolerance, max err {float((got - want).abs().max())}"


@pytest.mark.parametrize("B", [1, 64, 135, 333])
@pytest.mark.parametrize("layer", LAYERS, ids=[f"G{g}F{f}L{l}" for g, f, l in LAYERS])
def test_forward_and_both_gradients(layer, B):
    from haste_b200 import ffi
    G, F, L = layer
    D = 200
    inp = fo.make_inputs(B, D, L, F, G, 1, 1.1, seed=B + L, x_kind="normal", bias_zero=False)
    dev = {k: v.cuda() for k, v in inp.items()}
    xt = ffi.transpose_padded(dev["X"])
    assert torch.equal(xt[:, :B].cpu(), inp["X"].t()) and not xt[:, B:].any()
    z = ffi.forward(dev["loc"], xt, dev["W"], dev["bias"], G, B=B)
    _close(z, fo.forward(inp["loc"], inp["X"], inp["W"], inp["bias"], G, round_bf16=False), "logits")
    dY = (torch.randn(B, L, generator=torch.Generator().manual_seed(3)) * 0.5).to(torch.bfloat16)
    want_x, want_w = fo.backward_features(inp["loc"], inp["W"], dY, G, D), fo.backward_weights(inp["loc"], inp["X"], dY, G, L, round_bf16=False)
    dxt, dw, db = ffi.backward_both(xt, dev["W"], dev["loc"], dY.cuda(), G, B=B)
    for got_x, got_w, got_b in ((dxt, dw, db), (ffi.backward_features(xt, dev["W"], dev["loc"], dY.cuda(), G, B=B),
                                                *ffi.backward_weights(xt, dev["W"], dev["loc"], dY.cuda(), G, want_dbias=True, B=B))):
        _close(got_x, want_x, "dXt")
        _close(got_w, want_w, "dW")
        _close(got_b, dY.float().sum(0), "dbias")


@pytest.mark.parametrize("B", [8, 100, 333])
@pytest.mark.parametrize("loss", ["bce", "squared_hinge"])
@pytest.mark.parametrize("layer", LAYERS, ids=[f"G{g}F{f}L{l}" for g, f, l in LAYERS])
def test_step(layer, loss, B):
    """avg_pos 40 on few labels fills the tiles' target bitmaps, on many labels most groups take the entry list."""
    from haste_b200.fused import FusedFFIShard
    G, F, L = layer
    D, scale, lr, wd = 264, 0.5, 0.05, 1e-4
    inp = fo.make_inputs(B, D, L, F, G, min(40, max(1, L // 10)), 1.1, seed=B + L, x_kind="normal", bias_zero=False)
    kind = fo.LOSS_SQHINGE if loss == "squared_hinge" else fo.LOSS_BCE
    for mu, rng in ((0.0, "packed"), (0.0, "reference"), (0.9, "packed")):
        sh = FusedFFIShard(inp["loc"].cuda(), inp["W"].clone().cuda(), inp["bias"].clone().cuda(), G, D, loss=loss, lr=lr, weight_decay=wd,
                           momentum=mu, seed=42, rng=rng, grad_scale=scale)
        dxt, loss_dev = sh.step(inp["X"].cuda(), inp["targets"].cuda())
        ref = fo.train_step(inp["loc"], inp["X"], inp["W"], inp["bias"], inp["targets"], G, kind, lr, wd, 42, grad_scale=scale, rng_mode=rng)
        assert abs(float(loss_dev) - ref["loss"]) <= 2e-3 * abs(ref["loss"]) + 1e-3
        _close(dxt, ref["dXt"], "dXt")
        if mu == 0.0:
            same = (fo._bf16_to_bits(sh.w.cpu()) == fo._bf16_to_bits(ref["W_new"])).mean()
            assert same >= 0.95, f"{same:.3f} of the weights match bit for bit"
            _close(sh.bias, ref["bias_new"], "bias")
        else:
            _close(sh.mom_w, ref["dW"].float() + wd * inp["W"].float(), "momentum")
            _close(sh.mom_b, ref["dbias"].float() + wd * inp["bias"].float(), "bias momentum")
            _close(sh.w, inp["W"].float() - lr * sh.mom_w.cpu(), "weights")


@pytest.mark.parametrize("layer", [(32, 32, 32 * 5), (32, 64, 32 * 5), (32, 128, 32 * 5), (64, 64, 64 * 3), (128, 64, 128 * 3), (64, 128, 64 * 3)])
def test_step_bce_gradient_of_very_negative_logits(layer):
    """Logits around -12: the gradient is sigmoid(z) = 6e-6 and its sum over the batch has to be right to bf16, which an
    absolute error of the sigmoid would destroy (batch 100: the shapes and sizes that compute it with exp)."""
    from haste_b200.fused import FusedFFIShard
    G, F, L = layer
    B, D = 100, 264
    inp = fo.make_inputs(B, D, L, F, G, 1, 1.1, seed=5, x_kind="l2norm", bias_zero=True)
    inp["bias"] -= 12.0
    sh = FusedFFIShard(inp["loc"].cuda(), inp["W"].clone().cuda(), inp["bias"].clone().cuda(), G, D, loss="bce", lr=0.0, momentum=0.9, seed=1)
    sh.step(inp["X"].cuda(), torch.zeros(0, 2, dtype=torch.int32, device="cuda"))
    z = fo.forward(inp["loc"], inp["X"], inp["W"], inp["bias"], G).double()
    want = torch.sigmoid(z).sum(0)
    assert ((sh.mom_b.cpu().double() - want).abs() <= 2 ** -7 * want).all()          # two bf16 roundings of dY and its sum


@pytest.mark.parametrize("B,D", [(1, 1), (33, 70), (64, 768)])
def test_fp32_activations_are_cast_on_the_way(B, D):
    from haste_b200 import ffi
    x = torch.randn(B, D, generator=torch.Generator().manual_seed(1)).cuda()
    assert torch.equal(ffi.transpose_padded(x, f32=True), ffi.transpose_padded(x.to(torch.bfloat16)))
    dxt = x.t().contiguous()
    assert torch.equal(ffi.dxt_to_dx_sr(dxt, 7, torch.float32), ffi.dxt_to_dx_sr(dxt, 7).float())
    with pytest.raises(RuntimeError):
        ffi.transpose_padded(x)


@pytest.mark.parametrize("kind", ["near", "equal", "nan", "big_index"])
def test_rewire_scores_that_one_integer_does_not_order(kind):
    """Scores that agree in their upper 25 bits (near: they differ below; equal), NaN scores, and index tables with values
    beyond 24 bits: the kernel then compares the scores and indices themselves."""
    from haste_b200 import ffi
    D, L, F, G, frac = 1 << (26 if kind == "big_index" else 9), 300, 64, 64, 0.3
    gen = torch.Generator().manual_seed(3)
    W = torch.full((L, F), 0.5, dtype=torch.bfloat16)
    if kind == "near":
        for l0 in range(0, L, G):
            W[l0] = (2.0 ** -9 * (1 + torch.randperm(128, generator=gen)[:F] / 128.0)).to(torch.bfloat16)
    elif kind == "nan":
        W[::17, ::5] = float("nan")
    elif kind == "big_index":
        W = (torch.rand(L, F, generator=gen) - 0.5).to(torch.bfloat16)
    NG = (L + G - 1) // G
    loc0 = torch.randint(0, D, (NG, F), generator=gen, dtype=torch.int32)
    w, loc = W.clone().cuda(), loc0.clone().cuda()
    ffi.rewire(w, loc, None, D, G, 0, 1, 0.0, int(F * frac), 0, 0, True, 5, 1)
    if kind == "nan":      # a NaN score compares with nothing, so its rank is 0 and its slot is pruned
        want_zero = torch.stack([torch.isnan(W[g * G:(g + 1) * G].float()).any(0) for g in range(NG)])
        zero = torch.stack([(w.cpu()[g * G:(g + 1) * G].float() == 0).all(0) for g in range(NG)])
        assert not torch.isnan(w.float()).any() and (zero.sum(1) >= want_zero.sum(1)).all()
        return
    W1, loc1, _ = fo.rewire(W, loc0, G, D, "fraction", frac, None, init_mode="zero", regrow="replace", regroup=True, seed=5, step=1)
    assert torch.equal(loc.cpu(), loc1) and torch.equal(w.cpu(), W1)


# ------------------------------------------------------------------------------------------------ filtered top-k
def _check_topk(vals, idx, z, k, label0):
    """Against the full logits z (float, -inf and NaN never selected): values, and ids that are distinct, point at a logit
    of their value and stand in label order among equal values.  A logit may be the bf16 neighbour of z's (fp32 sum in
    another order)."""
    L = z.shape[1]
    z = torch.where(torch.isnan(z), torch.full_like(z, float("-inf")), z)
    want = torch.topk(z, min(k, L), dim=1).values
    got = vals[:, :want.shape[1]]
    none = torch.isinf(want) & (want < 0)
    assert torch.equal(torch.isinf(got) & (got < 0), none)
    assert (idx[:, :want.shape[1]][none] == -1).all() and (idx[:, want.shape[1]:] == -1).all() and torch.isinf(vals[:, want.shape[1]:]).all()
    ok = ~none
    if none.all():
        return
    near = (got - want).abs() <= 2 ** -7 * want.abs() + 1e-6
    assert near[ok].all() and (got == want)[ok].float().mean() >= 0.99
    ids = (idx[:, :want.shape[1]].long() - label0)
    assert ((ids >= 0) & (ids < L))[ok].all()
    at = torch.gather(z, 1, ids.clamp(0, L - 1))
    assert ((at - got).abs() <= 2 ** -7 * got.abs() + 1e-6)[ok].all() and (at == got)[ok].float().mean() >= 0.99
    for r, o in zip(ids.cpu(), ok.cpu()):
        assert len(set(r[o].tolist())) == int(o.sum())
    eq = (got[:, 1:] == got[:, :-1]) & ok[:, 1:]
    assert (ids[:, 1:] > ids[:, :-1])[eq].all()


@pytest.mark.parametrize("cfg", [
    dict(B=1, L=131073, F=128, G=64, k=5), dict(B=1, L=40, F=16, G=16, k=128), dict(B=3, L=5000, F=32, G=32, k=100),
    dict(B=8, L=70001, F=64, G=128, k=50), dict(B=7, L=300007, F=32, G=32, k=128),
    dict(B=9, L=16385, F=32, G=32, k=10), dict(B=40, L=160001, F=32, G=32, k=100), dict(B=200, L=40003, F=64, G=128, k=100),
    dict(B=130, L=30000, F=128, G=64, k=1), dict(B=17, L=20011, F=64, G=64, k=128), dict(B=16, L=20011, F=64, G=32, k=7), dict(B=16, L=20011, F=128, G=32, k=20),
], ids=lambda c: "-".join(f"{n}{v}" for n, v in c.items()))
def test_topk_fused(cfg):
    from haste_b200 import ffi
    from haste_b200.infer import ffi_topk
    B, L, F, G, k, D = cfg["B"], cfg["L"], cfg["F"], cfg["G"], cfg["k"], 256
    inp = fo.make_inputs(B, D, L, F, G, 1, 1.1, seed=11, x_kind="normal", bias_zero=False)
    dev = {n: v.cuda() for n, v in inp.items()}
    vals, idx = ffi_topk(dev["loc"], dev["W"], dev["bias"], dev["X"], k, G, label0=5)
    z = ffi.forward(dev["loc"], ffi.transpose_padded(dev["X"]), dev["W"], dev["bias"], G, B=B).float()
    _check_topk(vals, idx, z, k, 5)


@pytest.mark.parametrize("kind", ["ascending", "equal", "masked", "none"])
@pytest.mark.parametrize("B", [2, 16])
def test_topk_fused_unusual_logits(kind, B):
    """ascending: every later label beats all earlier ones, so the candidate lists overflow and the rows are computed
    again; equal: only the label id decides; masked: -inf and NaN biases are never selected; none: nothing is."""
    from haste_b200 import ffi
    from haste_b200.infer import ffi_topk
    D, L, F, G, k = 128, 16384 + 12007, 64, 64, 100
    inp = fo.make_inputs(B, D, L, F, G, 1, 1.1, seed=12, x_kind="normal", bias_zero=True)
    if kind == "ascending":
        inp["bias"] = (torch.arange(L) / 64.0).to(torch.bfloat16)
    elif kind == "equal":
        inp["W"].zero_()
    elif kind == "masked":
        inp["bias"][::3] = float("-inf")
        inp["bias"][1::3] = float("nan")
    else:
        inp["bias"][:] = float("-inf")
    dev = {n: v.cuda() for n, v in inp.items()}
    vals, idx = ffi_topk(dev["loc"], dev["W"], dev["bias"], dev["X"], k, G)
    z = ffi.forward(dev["loc"], ffi.transpose_padded(dev["X"]), dev["W"], dev["bias"], G, B=B).float()
    _check_topk(vals, idx, z, k, 0)
    if kind == "equal":
        assert torch.equal(idx.cpu(), torch.arange(k, dtype=torch.int32).expand(B, k))


SHAPES = [(32, 32), (32, 64), (64, 64), (32, 128), (128, 64), (64, 128)]


@pytest.mark.parametrize("mask", [float("-inf"), -3.0e38, -1.0e4])
@pytest.mark.parametrize("B", [100, 128])
@pytest.mark.parametrize("loss", ["bce", "squared_hinge"])
@pytest.mark.parametrize("G,F", SHAPES)
def test_step_with_masked_labels(G, F, loss, B, mask):
    """A label masked by a very negative bias adds nothing to the loss and to dX and keeps its weights bit for bit, also where
    the last batch tile has rows beyond the batch (their logits are the biases alone)."""
    from haste_b200.fused import FusedFFIShard
    D, L, scale = 264, 3 * G + 7, 0.5
    inp = fo.make_inputs(B, D, L, F, G, 3, 1.1, seed=B + F, x_kind="normal", bias_zero=False)
    masked = torch.zeros(L, dtype=torch.bool)
    masked[::7] = True
    targets = inp["targets"][~masked[inp["targets"][:, 1].long()]].contiguous()
    z = fo.forward(inp["loc"], inp["X"], inp["W"], inp["bias"], G).double()
    y = torch.zeros(B, L, dtype=torch.float64)
    y[targets[:, 0].long(), targets[:, 1].long()] = 1.0
    if loss == "bce":
        term, dY = torch.nn.functional.softplus(z) - y * z, torch.sigmoid(z) - y
    else:
        s = 2.0 * y - 1.0
        m = (1.0 - s * z).clamp_min(0.0)
        term, dY = m * m, -2.0 * s * m
    term[:, masked], dY[:, masked] = 0.0, 0.0
    want_loss, dY = float(term.sum()) * scale, (dY * scale).to(torch.bfloat16)
    bias = inp["bias"].clone()
    bias[masked] = mask
    want_x = fo.backward_features(inp["loc"], inp["W"], dY, G, D)
    for with_loss in (True, False):
        sh = FusedFFIShard(inp["loc"].cuda(), inp["W"].clone().cuda(), bias.clone().cuda(), G, D, loss=loss, lr=0.05, seed=42, grad_scale=scale)
        dxt, loss_dev = sh.step(inp["X"].cuda(), targets.cuda(), want_loss=with_loss)
        # as test_step: the logits are bf16, some one rounding away from the oracle's
        assert not with_loss or abs(float(loss_dev) - want_loss) <= 2e-3 * want_loss
        _close(dxt, want_x, "dXt")
        assert (fo._bf16_to_bits(sh.w.cpu()[masked]) == fo._bf16_to_bits(inp["W"][masked])).all()
        if mask != float("-inf"):          # (an infinite bias does not survive an update: 0 * inf in the weight decay)
            assert (fo._bf16_to_bits(sh.bias.cpu()[masked]) == fo._bf16_to_bits(bias[masked])).all()
        assert not torch.equal(sh.w.cpu()[~masked], inp["W"][~masked])


@pytest.mark.parametrize("loss", ["bce", "squared_hinge"])
@pytest.mark.parametrize("G,F", SHAPES)
def test_step_rows_beyond_the_batch_never_reach_the_gradients(G, F, loss):
    """Infinite weights and biases give those rows logits that are not finite.  Weight gradients are sums over the batch's rows
    alone: with B = 1 and finite loss gradients they stay finite, and an infinite one stays infinite."""
    from haste_b200.fused import FusedFFIShard
    B, D, L = 1, 264, 3 * G + 7
    inp = fo.make_inputs(B, D, L, F, G, 1, 1.1, seed=2, x_kind="relu", bias_zero=False)
    inp["X"] += 0.25                                        # positive: an infinite weight gives an infinite logit, not a NaN
    inp["W"][5, 3], inp["W"][G, 1] = float("-inf"), float("-inf")
    inp["bias"][9] = float("inf")
    sh = FusedFFIShard(inp["loc"].cuda(), inp["W"].clone().cuda(), inp["bias"].clone().cuda(), G, D, loss=loss, lr=0.05, momentum=0.9, seed=3)
    sh.step(inp["X"].cuda(), torch.zeros(0, 2, dtype=torch.int32, device="cuda"))
    mom_w, mom_b = sh.mom_w.cpu(), sh.mom_b.cpu()           # gradients (weight decay 0 leaves a NaN where the weight is infinite)
    at = torch.isinf(inp["W"].float())
    assert torch.isfinite(mom_w[[5, G]][~at[[5, G]]]).all() and (mom_b[[5, G]] == 0).all()
    if loss == "squared_hinge":
        assert torch.isinf(mom_w[9]).all()
    else:
        assert torch.isfinite(mom_w[9]).all()
    rest = torch.ones(L, dtype=torch.bool)
    rest[[5, G, 9]] = False
    assert torch.isfinite(mom_w[rest]).all() and torch.isfinite(mom_b[rest]).all()


@pytest.mark.parametrize("scale", [0.0, -0.5, 1e-22, 1e-9, 2.0 ** 40])
@pytest.mark.parametrize("G,F", [(32, 32), (128, 64)])
def test_hinge_step_with_any_gradient_scale(G, F, scale):
    """The scale multiplies loss and gradients, also where its square leaves fp32 or it is not positive."""
    from haste_b200.fused import FusedFFIShard
    B, D, L = 100, 264, 3 * G + 7
    inp = fo.make_inputs(B, D, L, F, G, 3, 1.1, seed=9, x_kind="normal", bias_zero=False)
    ref = fo.train_step(inp["loc"], inp["X"], inp["W"], inp["bias"], inp["targets"], G, fo.LOSS_SQHINGE, 0.0, 0.0, 42)
    sh = FusedFFIShard(inp["loc"].cuda(), inp["W"].clone().cuda(), inp["bias"].clone().cuda(), G, D, loss="squared_hinge", lr=0.0, seed=42,
                       grad_scale=scale)
    dxt, loss_dev = sh.step(inp["X"].cuda(), inp["targets"].cuda())
    assert abs(float(loss_dev) - ref["loss"] * scale) <= 2e-3 * abs(ref["loss"] * scale)
    want = ref["dXt"].double() * scale
    assert float((dxt.cpu().double() - want).norm()) <= 1e-2 * float(want.norm())


@pytest.mark.parametrize("L", [20011, 18944 * 9 + 70])
@pytest.mark.parametrize("G,F", SHAPES)
def test_topk_fused_ties_and_any_label_order(G, F, L):
    """The filtered path samples every n-th label tile.  equal: the label id alone decides, whichever launch a label belongs to;
    rising, falling: the best labels lie at one end; other_tiles: every label outside the sample beats the sample, so that the
    candidate lists overflow (more than 8192 labels) and the rows are computed again."""
    from haste_b200 import ffi
    from haste_b200.infer import ffi_topk
    B, D, k = 9, 128, 100
    tile = 64 if G == 32 and F < 128 else G
    inp = fo.make_inputs(B, D, L, F, G, 1, 1.1, seed=12, x_kind="normal", bias_zero=True)
    dev = {n: v.cuda() for n, v in inp.items()}
    x = dev["X"]
    ramp = torch.arange(L, device="cuda").float()
    n = 3 if L < 40000 else 12                    # the sample: every n-th tile
    for kind, bias in (("equal", torch.zeros_like(ramp)), ("rising", ramp / L * 8), ("falling", -ramp / L * 8),
                       ("other_tiles", 4.0 * (torch.arange(L, device="cuda") // tile % n != 0))):
        bias = bias.to(torch.bfloat16)
        features = torch.zeros_like(x) if kind == "equal" else x
        vals, idx = ffi_topk(dev["loc"], dev["W"], bias, features, k, G, label0=3)
        z = ffi.forward(dev["loc"], ffi.transpose_padded(features), dev["W"], bias, G, B=B).float()
        _check_topk(vals, idx, z, k, 3)
        if kind == "equal":
            assert torch.equal(idx.cpu(), (3 + torch.arange(k, dtype=torch.int32)).expand(B, k))


def test_topk_cost_does_not_depend_on_the_label_order():
    """Biases that rise with the label id, a first 16 K labels that are masked, a block of labels ahead of all others: the call takes
    about as long as with biases in random order.  (A bar set by the first labels made these 20 to 50 times slower.)"""
    from haste_b200.infer import ffi_topk
    B, D, L, F, G, k = 256, 768, 300007, 64, 128, 100
    inp = fo.make_inputs(B, D, L, F, G, 1, 1.1, seed=12, x_kind="l2norm", bias_zero=True)
    dev = {n: v.cuda() for n, v in inp.items()}
    random = torch.rand(L, generator=torch.Generator().manual_seed(1)) * 0.05
    masked, block = random.clone(), random.clone()
    masked[:16384] = float("-inf")
    block[100000:130000] += 1.0

    def ms(bias):
        bias = bias.to(torch.bfloat16).cuda()
        best = float("inf")
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ffi_topk(dev["loc"], dev["W"], bias, dev["X"], k, G)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    base = ms(random)
    for name, bias in (("rising", torch.sort(random).values), ("masked", masked), ("block", block)):
        assert ms(bias) <= 4.0 * base, name


def test_topk_of_a_batch_larger_than_a_slice():
    """Batches beyond 4096 rows go through in slices that share their scratch."""
    from haste_b200 import ffi
    from haste_b200.infer import ffi_topk
    B, D, L, F, G, k = 8201, 64, 20011, 32, 32, 10
    inp = fo.make_inputs(B, D, L, F, G, 1, 1.1, seed=5, x_kind="normal", bias_zero=False)
    dev = {n: v.cuda() for n, v in inp.items()}
    vals, idx = ffi_topk(dev["loc"], dev["W"], dev["bias"], dev["X"], k, G)
    z = ffi.forward(dev["loc"], ffi.transpose_padded(dev["X"]), dev["W"], dev["bias"], G, B=B).float()
    _check_topk(vals, idx, z, k, 0)
    from haste_b200._lib import lib
    n = [lib.haste_ffi_topk_fused_scratch(b, 768, 64, 670091, 128, 100) for b in (512, 4096, 8192, 20000)]
    assert n[0] < n[1] == n[2] == n[3] < 410 << 20


# ------------------------------------------------------------------------------------------------ accuracy and variants
@pytest.mark.parametrize("G,F", SHAPES)
def test_step_bce_gradient_accuracy_at_a_multiple_of_8(G, F):
    """Logits around -12 again, at the batch sizes where (128, 64) and (64, 128) take the sigmoid from tanh.approx: an absolute
    error of up to 2^-12 per logit there (half of the instruction's 2^-11), a relative one elsewhere."""
    from haste_b200.fused import FusedFFIShard
    B, D, L = 104, 264, 3 * G
    inp = fo.make_inputs(B, D, L, F, G, 1, 1.1, seed=5, x_kind="l2norm", bias_zero=True)
    inp["bias"] -= 12.0
    sh = FusedFFIShard(inp["loc"].cuda(), inp["W"].clone().cuda(), inp["bias"].clone().cuda(), G, D, loss="bce", lr=0.0, momentum=0.9, seed=1)
    sh.step(inp["X"].cuda(), torch.zeros(0, 2, dtype=torch.int32, device="cuda"))
    z = fo.forward(inp["loc"], inp["X"], inp["W"], inp["bias"], G).double()
    want = torch.sigmoid(z).sum(0)
    tanh = G * F == 128 * 64
    assert ((sh.mom_b.cpu().double() - want).abs() <= 2 ** -7 * want + (B * 2.0 ** -12 if tanh else 0.0)).all()


def test_rewire_prunes_the_slots_with_nan_scores_and_the_lowest_others():
    """A NaN compares with nothing: its slot has rank 0 and is pruned, and the other slots' ranks do not count it."""
    from haste_b200 import ffi
    D, L, F, G, n_prune = 512, 300, 64, 64, 19
    gen = torch.Generator().manual_seed(3)
    W = (torch.rand(L, F, generator=gen) - 0.5).to(torch.bfloat16)
    W[::17, ::5] = float("nan")
    NG = (L + G - 1) // G
    loc0 = torch.stack([torch.randperm(D, generator=gen)[:F] for _ in range(NG)]).to(torch.int32)
    w, loc = W.clone().cuda(), loc0.clone().cuda()
    ffi.rewire(w, loc, None, D, G, 0, 1, 0.0, n_prune, 1, 0, False, 5, 1)
    for g in range(NG):
        rows = W[g * G:(g + 1) * G].float()
        score = torch.zeros(F)
        for r in rows:                                        # fp32, one row after the other, as the kernel sums
            score = score + r.abs()
        score = score / rows.shape[0]
        ahead = (score[None, :] < score[:, None]) | ((score[None, :] == score[:, None]) & (torch.arange(F)[None, :] < torch.arange(F)[:, None]))
        pruned = ahead.sum(1) < n_prune
        got = w[g * G:(g + 1) * G].cpu()
        assert (got[:, pruned] == 0).all()
        assert torch.equal(got[:, ~pruned], W[g * G:(g + 1) * G][:, ~pruned])
        assert torch.equal(loc[g].cpu()[~pruned], loc0[g][~pruned])
        assert len(set(loc[g].tolist())) == F                 # 'unused' regrowth


@pytest.mark.parametrize("rng", ["reference", "packed"])
@pytest.mark.parametrize("G,F,L", [(64, 64, 64 * 160 + 33), (32, 64, 32 * 7), (32, 64, 32 * 310 + 1), (32, 128, 32 * 160 + 9), (32, 32, 32 * 401 + 7)])
def test_update_variant_of_the_backward(G, F, L, rng):
    """Backward-weights fused with the update against the unfused kernel and the oracle's update, bit for bit."""
    import numpy as np
    from haste_b200 import ffi
    B, D, label0, seed, step, lr, wd = 136, 200, 640, 123, 4, 0.05, 1e-4
    inp = fo.make_inputs(B, D, L, F, G, 1, 1.1, seed=L, x_kind="normal", bias_zero=False)
    dev = {k: v.cuda() for k, v in inp.items()}
    xt = ffi.transpose_bf16(dev["X"])
    gen = torch.Generator().manual_seed(2)
    dY = (torch.randn(B, L, generator=gen) * 0.3).to(torch.bfloat16).cuda()
    dw, db = ffi.backward_weights(xt, dev["W"], dev["loc"], dY, G, want_dbias=True)
    for mu in (0.0, 0.9):
        mom, momb = torch.randn(L, F, generator=gen) * 0.01, torch.randn(L, generator=gen) * 0.01
        want_w, want_m = fo.sgd_update(inp["W"], dw.cpu(), mom, lr, wd, mu, True, True, fo.rand16_for((L, F), seed, step, rng, label0))
        want_b, want_mb = fo.sgd_update(inp["bias"], db.cpu(), momb, lr, wd, mu, True, True,
                                        fo.rand16_for((L, 1), seed, step, rng, label0, is_bias=True).reshape(L))
        w, b, m, mb = dev["W"].clone(), dev["bias"].clone(), mom.clone().cuda(), momb.clone().cuda()
        ffi.bww_sr_sgd(xt, dev["loc"], dY, w, b, m, mb, G, label0, lr, wd, mu, seed, step, ffi.make_flags(sr=True, contract=True, rng=rng))
        assert np.array_equal(fo._bf16_to_bits(w.cpu()), fo._bf16_to_bits(want_w)) and np.array_equal(fo._bf16_to_bits(b.cpu()), fo._bf16_to_bits(want_b))
        if mu:
            assert torch.equal(m.cpu(), want_m) and torch.equal(mb.cpu(), want_mb)


@pytest.mark.parametrize("G,F", SHAPES)
def test_step_on_fewer_ctas(G, F):
    """set_max_ctas: the same weights and bias, in a time that shows that the limit holds."""
    from haste_b200 import _lib
    from haste_b200.fused import FusedFFIShard
    B, D, L = 104, 264, G * 592 + 5                           # at least two tiles for each of 148 CTAs
    inp = fo.make_inputs(B, D, L, F, G, 3, 1.1, seed=4, x_kind="l2norm", bias_zero=False)
    x, t = inp["X"].cuda(), inp["targets"].cuda()

    def run():
        sh = FusedFFIShard(inp["loc"].cuda(), inp["W"].clone().cuda(), inp["bias"].clone().cuda(), G, D, loss="bce", lr=0.05, seed=42)
        sh.step(x, t)
        w, b = sh.w.clone(), sh.bias.clone()
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        for _ in range(5):
            sh.step(x, t)
        end.record()
        end.synchronize()
        return w, b, start.elapsed_time(end)

    want_w, want_b, base = run()
    try:
        _lib.check(_lib.lib.haste_ffi_set_max_ctas(3), "set_max_ctas")
        w, b, few = run()
    finally:
        _lib.check(_lib.lib.haste_ffi_set_max_ctas(0), "set_max_ctas")
    assert torch.equal(w, want_w) and torch.equal(b, want_b)
    assert few >= 3.0 * base


@pytest.mark.parametrize("L", [18944 * 9 + 70, 18944 + 1, 200])
@pytest.mark.parametrize("G,F", SHAPES)
def test_topk_fused_sees_every_tile(G, F, L):
    """One label of every tile in turn is the best there is: the sample and the filter launches together hold each tile once."""
    from haste_b200.infer import ffi_topk
    B, D, tile, k = 9, 16 * F, 64 if G == 32 and F < 128 else G, 128
    loc = torch.arange((L + G - 1) // G * F, dtype=torch.int32, device="cuda").reshape(-1, F) % D
    W, x = torch.zeros(L, F, dtype=torch.bfloat16, device="cuda"), torch.ones(B, D, dtype=torch.bfloat16, device="cuda")
    for t0 in range(0, (L + tile - 1) // tile, k):
        best = torch.arange(t0, min(t0 + k, (L + tile - 1) // tile)) * tile
        best = torch.minimum(best + (best * 7 // tile) % tile, torch.tensor(L - 1))
        bias = torch.zeros(L, dtype=torch.bfloat16)
        bias[best] = 1.0
        vals, idx = ffi_topk(loc, W, bias.cuda(), x, len(best), G)
        assert torch.equal(idx.cpu(), best.to(torch.int32).expand(B, -1)) and (vals == 1.0).all()
