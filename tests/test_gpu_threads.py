"""The tensor-core paths as the first CUDA work of a thread: its results are the main thread's."""
import threading

import pytest
import torch

from pragnosia_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("delta", [False, True])
@pytest.mark.parametrize("what", ["forward", "gradients", "linear"])
def test_first_work_of_a_thread(what, delta):
    x = synth.assoc_op_inputs(1, 2, 130, 64, seed=1, delta=True, with_state=True)
    q, k, v = (x[n].cuda().bfloat16() for n in "qkv")
    la, beta = x["la"].cuda(), x["beta"].cuda() if delta else None
    W = torch.eye(64, device="cuda").bfloat16()
    kept = ops.scan_train_fwd(q, k, v, la, beta)

    def work():
        if what == "forward":
            return ops.prefill(q, k, v, la, beta)[:2]
        if what == "gradients":
            return ops.scan_train_bwd(q, k, v, la, beta, *kept[2:], q)[:4]
        return [ops.linear_act(q[0, 0], W, act=None), ops.batch_linear(q[0, 0, :16], W)]

    want, got = work(), []
    torch.cuda.synchronize()
    t = threading.Thread(target=lambda: got.append(work()))
    t.start(); t.join()
    torch.cuda.synchronize()
    assert got and all(torch.equal(a, b) for a, b in zip(got[0], want))
