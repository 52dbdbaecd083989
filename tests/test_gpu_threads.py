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


@pytest.mark.parametrize("D", [64, 128])
def test_fp32_calls_of_two_sizes_at_once(D):
    """Two threads, each on a stream of its own: the output kernel of few chunks is launched with more shared memory than that of
    many, and neither launch may depend on which size came to the function last. Results to the bit, none missing."""
    sizes, n = ((1, 2, 512), (8, 12, 512)), 3000
    args = []
    for i, (B, H, T) in enumerate(sizes):
        x = synth.assoc_op_inputs(B, H, T, D, seed=i, with_state=True)
        args.append([x[s].cuda() for s in ("q", "k", "v", "la", "S0")])
    call = lambda a: ops.prefill(a[0], a[1], a[2], a[3], None, S0=a[4])[:2]
    want = [call(a) for a in args]
    torch.cuda.synchronize()
    off, errors = [torch.zeros((), dtype=torch.long, device="cuda") for _ in sizes], []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(n):
                    for a, b in zip(call(args[i]), want[i]):
                        off[i] += (a != b).any()
                torch.cuda.current_stream().synchronize()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads: t.start()
    for t in threads: t.join()
    torch.cuda.synchronize()
    assert not errors, errors[0]
    assert [int(o) for o in off] == [0, 0]
