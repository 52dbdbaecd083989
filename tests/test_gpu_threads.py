"""Threads: first CUDA work in one, calls of several sizes at once, what a refused call leaves behind."""
import ctypes
import threading

import pytest
import torch

from pragnosia_b200 import _lib, ops, synth

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


def test_a_refused_launch_leaves_no_error_behind():
    """A launch that the runtime refuses on the host (into a capture that is no longer valid) is that call's error alone: the thread's
    next call succeeds."""
    rt = ctypes.CDLL("libcudart.so.12")                              # the one torch has loaded
    x, w, z = (torch.ones(4, 64, device="cuda") for _ in range(3))
    torch.cuda.synchronize()
    bad, graph = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaStreamCreate(ctypes.byref(bad)) == 0
    call = lambda stream: _lib.lib().pgb_add_norm(*(ctypes.c_void_p(p) for p in (x.data_ptr(), 0, w.data_ptr(), 0)), ctypes.c_float(1e-6), 0,
                                                  None, ctypes.c_void_p(z.data_ptr()), ctypes.c_longlong(4), 64, 0, stream)
    assert call(None) == 0
    assert rt.cudaStreamBeginCapture(bad, 0) == 0
    assert rt.cudaDeviceSynchronize() != 0                           # not allowed meanwhile: the capture is lost
    assert call(bad) != 0
    assert rt.cudaStreamEndCapture(bad, ctypes.byref(graph)) != 0
    rt.cudaGetLastError()
    assert call(None) == 0
    torch.cuda.synchronize()
    assert rt.cudaStreamDestroy(bad) == 0
