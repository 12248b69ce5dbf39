"""Calls from several host threads, each on its own stream.  A kernel's dynamic shared memory limit belongs to the function and not
to a call, so a launch must not depend on what another thread's call of the same kernel needed."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import ffi_oracle as fo


def _run(calls, reps):
    errors = []

    def work(call):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(reps):
                    call()
                torch.cuda.current_stream().synchronize()
        except Exception as e:
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("B", [4, 64])
def test_topk_with_different_k(B):
    from haste_b200.infer import ffi_topk
    inp = fo.make_inputs(B, 256, 40000, 64, 128, 1, 1.1, seed=3, x_kind="normal", bias_zero=False)
    d = {n: v.cuda() for n, v in inp.items()}
    call = lambda k: ffi_topk(d["loc"], d["W"], d["bias"], d["X"], k, 128)
    want, got = call(128), {}
    _run([lambda k=k: got.__setitem__(k, call(k)) for k in (1, 5, 100, 128)], 2000)
    for k, (vals, idx) in got.items():
        assert torch.equal(vals, want[0][:, :k]) and torch.equal(idx, want[1][:, :k])


def test_step_with_different_label_counts():
    """The preparation kernel's counters: one word per label group."""
    from haste_b200.fused import FusedFFIShard
    calls = []
    for L, G in ((700000, 16), (300000, 16), (500, 16)):
        inp = fo.make_inputs(8, 64, L, 16, G, 3, 1.1, seed=3, x_kind="normal")
        sh = FusedFFIShard(inp["loc"].cuda(), inp["W"].cuda(), inp["bias"].cuda(), G, 64, seed=1)
        calls.append(lambda sh=sh, x=inp["X"].cuda(), t=inp["targets"].cuda(): sh.step(x, t))
    _run(calls, 1000)


def test_rewire_of_different_shapes():
    from haste_b200 import ffi
    calls = []
    for F, G in ((128, 128), (16, 16), (128, 64)):
        inp = fo.make_inputs(1, 256, 2000, F, G, 1, 1.1, seed=3, x_kind="normal")
        w, loc = inp["W"].cuda(), inp["loc"].cuda()
        calls.append(lambda w=w, loc=loc, G=G: ffi.rewire(w, loc, None, 256, G, 0, 1, 0.0, 3, 1, 0, True, 5, 1))
    _run(calls, 2000)
