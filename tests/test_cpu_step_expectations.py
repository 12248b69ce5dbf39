"""What the GPU test of the fused step's branches can see: a step that loses one label group's positives, or one positive, is outside each of
its tolerances.  (On the CPU: the mistake is planted in the expectation.)"""
import pytest
import torch

from test_gpu_step_paths import SHAPES, STEP_LR, STEP_SCALE, step_case, step_expected, step_tolerances


@pytest.mark.parametrize("loss", ["bce", "squared_hinge"])
@pytest.mark.parametrize("G,F", SHAPES)
def test_lost_positives_are_outside_every_tolerance(G, F, loss):
    inp = step_case(G, F, 61, False)
    want = step_expected(inp, G, loss, STEP_SCALE)
    tol_loss, tol_x, tol_w = step_tolerances(*want)
    label = inp["targets"][:, 1]
    lost = [label // G == g for g in label.div(G, rounding_mode="floor").unique()]
    last = torch.zeros_like(label, dtype=torch.bool)
    last[-1] = True
    for drop in lost + [last]:
        got_loss, got_x, got_w = step_expected(dict(inp, targets=inp["targets"][~drop]), G, loss, STEP_SCALE)
        assert abs(got_loss - want[0]) > tol_loss
        assert ((got_x - want[1]).abs() > tol_x).any()
        assert ((got_w - want[2]).abs() > tol_w).any()
        assert (STEP_LR * (got_w - want[2]).abs() > (inp["W"].float() - STEP_LR * want[2]).abs() / 128 + STEP_LR * tol_w + 1e-6).any()
