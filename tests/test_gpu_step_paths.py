"""GPU parity tests of the fused step's branches: few targets (put right after the plain loop, or by their bits) and many (bitmap) in the
label groups of one layer, targets at the edges of warps and tiles and listed twice, logits too large for the correction, and batch
sizes with 16-byte aligned and unaligned rows of dX."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import ffi_oracle as fo

SHAPES = [(32, 32), (32, 64), (64, 64), (32, 128), (128, 64), (64, 128)]


@pytest.mark.parametrize("B", [36, 61, 132])
@pytest.mark.parametrize("loss", ["bce", "squared_hinge"])
@pytest.mark.parametrize("G,F", SHAPES)
def test_step_targets_few_many_twice_and_large_logits(G, F, loss, B):
    from haste_b200.fused import FusedFFIShard
    D, L, scale, lr = 264, 7 * G + 5, 0.5, 0.05
    inp = fo.make_inputs(B, D, L, F, G, 1, 1.1, seed=B + F, x_kind="normal", bias_zero=False)
    bias = inp["bias"].clone()
    bias[2 * G + 3], bias[2 * G + 4] = 3000.0, -3000.0          # beyond what a difference of two losses can carry
    rows = [0, 31, 32 % B, min(63, B - 1), B - 1]
    pairs = [(r, c) for r in rows for c in (0,)]                                              # group 0: the first label in the edge rows
    pairs += [(0, G + G - 1), (0, G + G - 1), (B - 1, G), (B - 1, G), (B - 1, G + 15)]          # group 1: the last label twice, the first twice
    pairs += [(1, 2 * G + 3), (2, 2 * G + 4), (3, 2 * G + 5)]                                 # group 2: large logits as positives
    pairs += [(r % B, 3 * G + (5 * r) % G) for r in range(40)]                                # group 3: more than the entry list holds
    pairs += [(0, 7 * G + 4), (B - 1, 7 * G)]                                                 # the ragged last group
    pairs += [(r % B, 5 * G + r) for r in range(8)]                                           # group 5: exactly a full list
    targets = torch.tensor(pairs, dtype=torch.int32)
    z = fo.forward(inp["loc"], inp["X"], inp["W"], bias, G).double()
    y = torch.zeros(B, L, dtype=torch.float64)
    y[targets[:, 0].long(), targets[:, 1].long()] = 1.0
    if loss == "bce":
        term, dY = torch.nn.functional.softplus(z) - y * z, torch.sigmoid(z) - y
    else:
        s = 2.0 * y - 1.0
        m = (1.0 - s * z).clamp_min(0.0)
        term, dY = m * m, -2.0 * s * m
    want_loss, dY = float(term.sum()) * scale, (dY * scale).to(torch.bfloat16)
    want_x, want_w = fo.backward_features(inp["loc"], inp["W"], dY, G, D), fo.backward_weights(inp["loc"], inp["X"], dY, G, L, round_bf16=False)
    for mu in (0.0, 0.9):
        sh = FusedFFIShard(inp["loc"].cuda(), inp["W"].clone().cuda(), bias.clone().cuda(), G, D, loss=loss, lr=lr, momentum=mu, seed=42, grad_scale=scale)
        dxt, loss_dev = sh.step(inp["X"].cuda(), targets.cuda())
        # the logits are bf16, some one rounding away from the oracle's
        assert abs(float(loss_dev) - want_loss) <= 2e-3 * want_loss
        big = 1e-3 * max(1.0, float(want_x.abs().max())) + 1e-2 * want_x.abs()
        assert ((dxt.cpu() - want_x).abs() <= big).all()
        if mu == 0.0:
            # w' = w - lr g, stochastically rounded to bf16: one unit in the last place (2^-7) of w', and g as far off as dW may be
            want = inp["W"].float() - lr * want_w
            tol = want.abs() / 128 + lr * (1e-2 * want_w.abs() + 1e-3 * max(1.0, float(want_w.abs().max()))) + 1e-6
            assert ((sh.w.float().cpu() - want).abs() <= tol).all()
        else:
            tol = 1e-2 * want_w.abs() + 1e-3 * max(1.0, float(want_w.abs().max()))
            assert ((sh.mom_w.cpu() - want_w).abs() <= tol).all()


def step_case(G, F, B, large):
    """Inputs whose negatives have next to no hinge loss and little BCE loss (bias -3), so that every positive shows in the loss, in its batch row
    of dX and in its label's row of dW.  ``large``: two labels with logits near +-3000, positive for one row each, instead of the patterns."""
    D, L = 264, 7 * G + 5
    inp = fo.make_inputs(B, D, L, F, G, 1, 1.1, seed=B + F, x_kind="normal", bias_zero=False)
    inp["bias"] = (inp["bias"].float() - 3.0).to(torch.bfloat16)
    if large:
        inp["bias"][2 * G + 3], inp["bias"][2 * G + 4] = 3000.0, -3000.0        # beyond what a difference of two losses can carry
        pairs = [(1, 2 * G + 3), (2, 2 * G + 4), (3, 2 * G + 5)]
    else:
        rows = [0, 31, 32 % B, min(63, B - 1), B - 1]
        pairs = [(r, 0) for r in rows]                                                       # group 0: the first label in the edge rows
        pairs += [(0, G + G - 1), (0, G + G - 1), (B - 1, G), (B - 1, G), (B - 1, G + 15)]     # group 1: the last label twice, the first twice
        pairs += [(r % B, 3 * G + (5 * r) % G) for r in range(40)]                           # group 3: more than the entry list holds
        pairs += [(r, 4 * G + 7 * r) for r in range(4)]                                      # group 4: as many columns as are put right one by one
        pairs += [(r % B, 5 * G + r) for r in range(8)]                                      # group 5: exactly a full list
        pairs += [(r, 6 * G + 6 * r) for r in range(5)]                                      # group 6: a column more than in group 4
        pairs += [(0, 7 * G + 4), (B - 1, 7 * G)]                                            # the ragged last group
    inp["targets"] = torch.tensor(pairs, dtype=torch.int32)
    return inp


def step_expected(inp, G, loss, scale):
    """(loss, dxt, dW) of a step, from logits rounded to bf16 and in 64 bits from there; dY is bf16."""
    B, D = inp["X"].shape
    L = inp["W"].shape[0]
    z = fo.forward(inp["loc"], inp["X"], inp["W"], inp["bias"], G).double()
    y = torch.zeros(B, L, dtype=torch.float64)
    y[inp["targets"][:, 0].long(), inp["targets"][:, 1].long()] = 1.0
    if loss == "bce":
        term, dY = torch.nn.functional.softplus(z) - y * z, torch.sigmoid(z) - y
    else:
        s = 2.0 * y - 1.0
        m = (1.0 - s * z).clamp_min(0.0)
        term, dY = m * m, -2.0 * s * m
    dY = (dY * scale).to(torch.bfloat16)
    return (float(term.sum()) * scale, fo.backward_features(inp["loc"], inp["W"], dY, G, D),
            fo.backward_weights(inp["loc"], inp["X"], dY, G, L, round_bf16=False).float())


def step_tolerances(want_loss, want_x, want_w):
    """Some logits are one bf16 rounding (2^-8 of them at most) away from the oracle's, and so are their gradients.  That is seen against the other
    terms of the same sum: the batch row of dX (dxt is [D, B]), the label's row of dW.  A negative at the margin has a gradient of that
    size or none."""
    tol_x = 1e-2 * want_x.abs() + 1e-2 * want_x.abs().amax(0, keepdim=True) + 1e-3
    tol_w = 1e-2 * want_w.abs() + 1e-2 * want_w.abs().amax(1, keepdim=True) + 2e-2
    return 1e-4 * want_loss, tol_x, tol_w


STEP_SCALE, STEP_LR = 0.5, 0.05


@pytest.mark.parametrize("large", [False, True], ids=["patterns", "large-logits"])
@pytest.mark.parametrize("B", [36, 61, 132, 136])
@pytest.mark.parametrize("loss", ["bce", "squared_hinge"])
@pytest.mark.parametrize("G,F", SHAPES)
def test_step_positives_by_row_and_by_label(G, F, loss, B, large):
    from haste_b200.fused import FusedFFIShard
    inp = step_case(G, F, B, large)
    want_loss, want_x, want_w = step_expected(inp, G, loss, STEP_SCALE)
    tol_loss, tol_x, tol_w = step_tolerances(want_loss, want_x, want_w)
    if large:
        tol_loss = 2e-3 * want_loss                                  # the logits near 3000 may be one bf16 rounding away
    if loss == "bce" and G * F == 128 * 64 and B % 8 == 0:
        tol_loss += 2.0 ** -12 * B * inp["W"].shape[0] * STEP_SCALE     # the sigmoid comes from tanh.approx there, off by up to 2^-12
    for mu in (0.0, 0.9):
        sh = FusedFFIShard(inp["loc"].cuda(), inp["W"].clone().cuda(), inp["bias"].clone().cuda(), G, inp["X"].shape[1], loss=loss, lr=STEP_LR,
                           momentum=mu, seed=42, grad_scale=STEP_SCALE)
        dxt, loss_dev = sh.step(inp["X"].cuda(), inp["targets"].cuda())
        assert abs(float(loss_dev) - want_loss) <= tol_loss
        assert ((dxt.cpu() - want_x).abs() <= tol_x).all()
        if mu == 0.0:
            # w' = w - lr g, stochastically rounded to bf16: one unit in the last place (2^-7) of w', and g as far off as dW may be
            want = inp["W"].float() - STEP_LR * want_w
            assert ((sh.w.float().cpu() - want).abs() <= want.abs() / 128 + STEP_LR * tol_w + 1e-6).all()
        else:
            assert ((sh.mom_w.cpu() - want_w).abs() <= tol_w).all()


@pytest.mark.parametrize("off", [0, 1, 6])
@pytest.mark.parametrize("B,tail", [(128, 0), (129, 1), (256, 7), (300, 63)])
@pytest.mark.parametrize("G,F", SHAPES)
def test_backward_reads_dy_at_any_offset_and_nothing_else(G, F, B, tail, off):
    """The rows of dY are copied in aligned 16-byte chunks: all of them with one pointer away from the tensor's ends, chunk by chunk at the
    ends.  What lies before and after the gradient in memory is NaN here and must not be seen."""
    from haste_b200 import ffi
    D = 200
    full = fo.make_inputs(B, D, 3 * G + tail, F, G, 1, 1.1, seed=B, x_kind="normal", bias_zero=False)
    for L in (3 * G + tail, max(tail, 1)):
        inp = dict(loc=full["loc"][:(L + G - 1) // G].contiguous(), X=full["X"], W=full["W"][:L].contiguous())
        buf = torch.full((off + B * L + 16,), float("nan"), dtype=torch.bfloat16)
        buf[off:off + B * L] = (torch.randn(B * L, generator=torch.Generator().manual_seed(L)) * 0.5).to(torch.bfloat16)
        dev = {k: inp[k].cuda() for k in ("loc", "X", "W")}
        gbuf = buf.cuda()
        dY, dY_dev = buf[off:off + B * L].view(B, L), gbuf[off:off + B * L].view(B, L)
        dxt, dw, db = ffi.backward_both(ffi.transpose_padded(dev["X"]), dev["W"], dev["loc"], dY_dev, G, B=B)
        for got, want in ((dxt, fo.backward_features(inp["loc"], inp["W"], dY, G, D)),
                          (dw, fo.backward_weights(inp["loc"], inp["X"], dY, G, L, round_bf16=False)), (db, dY.float().sum(0))):
            got, want = got.float().cpu(), want.float()
            # bf16 outputs of fp32 sums
            assert ((got - want).abs() <= 1e-3 * max(1.0, float(want.abs().max())) + 1e-2 * want.abs()).all()


def hinge_loss_beside(G, F, z_pos):
    """(loss, what it should be, number of positives, scale).  A positive beyond the margin has no loss, however far.  Every negative lies on the margin but one per row and group, which is all there is
    to sum."""
    from haste_b200.fused import FusedFFIShard
    B, NG, D, scale = 64, 5, 160, 0.3
    L, gen = NG * G, torch.Generator().manual_seed(F)
    loc = torch.stack([torch.randperm(D, generator=gen)[:F].sort().values for _ in range(NG)]).int()
    X = torch.zeros(B, D, dtype=torch.bfloat16)
    X[torch.arange(B), torch.arange(B)] = 1.0                      # row b has feature b alone: weights set the logits one by one
    W, bias = torch.zeros(L, F, dtype=torch.bfloat16), torch.full((L,), -1.0, dtype=torch.bfloat16)
    pairs, n_off = [], 0
    for g in range(NG):
        slots = [k for k in range(F) if int(loc[g, k]) < B]
        for i in (0, 1):                                           # two rows with a positive and, in the same columns' half, a negative off the margin
            b, k = int(loc[g, slots[i]]), slots[i]
            W[g * G + 3 + i, k] = z_pos + 1.0                      # logit z_pos
            W[g * G + 9 + i, k] = 0.25                             # logit -0.75: loss 1/16
            pairs.append((b, g * G + 3 + i))
            n_off += 1
    z = fo.forward(loc, X, W, bias, G).double()
    assert float(z[pairs[0][0], pairs[0][1]]) == pytest.approx(z_pos, rel=2 ** -8)
    sh = FusedFFIShard(loc.cuda(), W.cuda(), bias.cuda(), G, D, loss="squared_hinge", lr=0.0, seed=1, grad_scale=scale)
    _, loss = sh.step(X.cuda(), torch.tensor(sorted(pairs), dtype=torch.int32).cuda())
    want = n_off / 16.0 * scale
    return float(loss), want, len(pairs), scale


@pytest.mark.parametrize("z_pos", [8.0, 50.0, 300.0, 900.0])
@pytest.mark.parametrize("G,F", SHAPES)
def test_hinge_loss_beside_confident_positives(G, F, z_pos):
    """Beside positives of z_pos the loss must come out to the accuracy of an fp32 sum."""
    loss, want, _, _ = hinge_loss_beside(G, F, z_pos)
    # ten equal terms, each rounded a few times to 2^-24
    assert abs(loss - want) <= 1e-5 * want


@pytest.mark.parametrize("z_pos", [1.0, 1.5, 3.0, 3.9375])
@pytest.mark.parametrize("G,F", SHAPES)
def test_hinge_loss_beside_positives_taken_out_again(G, F, z_pos):
    """Positives that may have been counted as negatives first, with (1 + z)^2, and taken out again: at most six roundings to 2^-24 of that
    each (a partial sum's other terms are 0 but one), beside those of the sum itself."""
    loss, want, n, scale = hinge_loss_beside(G, F, z_pos)
    assert abs(loss - want) <= 1e-5 * want + 6 * n * 2.0 ** -24 * (1.0 + z_pos) ** 2 * scale


@pytest.mark.parametrize("B,off", [(64, 0), (64, 1), (136, 3), (100, 6)])
@pytest.mark.parametrize("G,F", SHAPES)
def test_single_gradients_against_both_over_several_groups_a_cta(G, F, B, off):
    """The kernels that make one gradient, or update with it, have accumulator stages and copy loops of their own.  The sums are the same in the
    same order: dW, dbias and the updated weights bit for bit, dX up to the order of its reductions."""
    from haste_b200 import ffi
    D, L = 160, (5 if G == 128 or F == 128 else 9) * 148 * G // 2 + 3        # more than two tiles for most CTAs, the last one ragged
    gen = torch.Generator(device="cuda").manual_seed(B + F)
    loc = torch.rand((L + G - 1) // G, D, generator=gen, device="cuda").topk(F, dim=1).indices.sort(dim=1).values.int()
    W = ((torch.rand(L, F, generator=gen, device="cuda") * 2 - 1) / F ** 0.5).to(torch.bfloat16)
    bias = torch.randn(L, generator=gen, device="cuda").to(torch.bfloat16)
    X = torch.randn(B, D, generator=gen, device="cuda").to(torch.bfloat16)
    buf = torch.randn(off + B * L + 16, generator=gen, device="cuda").to(torch.bfloat16)
    dY, xt = buf[off:off + B * L].view(B, L), ffi.transpose_padded(X)
    dxt, dw, db = ffi.backward_both(xt, W, loc, dY, G, B=B)
    want = torch.zeros(B, D, device="cuda", dtype=torch.float64)
    for g0 in range(0, loc.shape[0], 256):                                   # dX[b, loc[g, k]] += sum over the group's labels of dY W
        for g in range(g0, min(g0 + 256, loc.shape[0])):
            rows = slice(g * G, min(g * G + G, L))
            want.index_add_(1, loc[g].long(), dY[:, rows].double() @ W[rows].double())
    # fp32 sums of L F / D label terms in any order
    tol = 2.0 ** -20 * (L * F / D) * float(dY.float().std() * W.float().std()) + 1e-5 * want.abs()
    for got in (dxt, ffi.backward_features(xt, W, loc, dY, G, B=B)):
        assert ((got[:, :B].t().double() - want).abs() <= tol).all()
    dw1, db1 = ffi.backward_weights(xt, W, loc, dY, G, want_dbias=True, B=B)
    assert torch.equal(dw1, dw) and torch.equal(db1, db)
    if B % 8 == 0:
        for rng in ("packed", "reference"):
            flags = ffi.make_flags(rng=rng)
            w1, b1, w2 = W.clone(), bias.clone(), W.clone()
            ffi.bww_sr_sgd(xt, loc, dY, w1, b1, None, None, G, 0, 0.05, 1e-4, 0.0, 7, 2, flags)
            ffi.sgd_sr_update(w2, dw, None, 0, 0.05, 1e-4, 0.0, 7, 2, flags)
            assert torch.equal(w1, w2)
