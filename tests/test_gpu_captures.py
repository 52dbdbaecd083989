"""Captured passes against what changes around them: caches that are outgrown, switches."""
import threading
import weakref

import pytest
import torch

from pragnosia_b200.generate import Decoder
from pragnosia_b200.model import LM

pytestmark = pytest.mark.gpu
torch.set_grad_enabled(False)
DEV = "cuda"


def lm(mixer, ctx=64, d=128, vocab=256, layers=2, seed=0):
    torch.manual_seed(seed)
    m = LM(vocab=vocab, d=d, layers=layers, mlp_mult=2, ctx=ctx, mixer=mixer, norm="rms")
    return m.to(DEV).to(torch.bfloat16).eval()


def ids(B, T, seed, vocab=256):
    return torch.randint(0, vocab, (B, T), device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed))


@pytest.mark.parametrize("mixer,d", [("aspin", 128), ("dspin", 128), ("hspin", 256), ("fspin", 128)])
@pytest.mark.parametrize("T", [64, 128, 150])
def test_a_graph_outlives_the_caches_it_read(mixer, d, T):
    """Window positions, rotation tables and positions are cached and replaced by longer ones: a graph captured before keeps its own."""
    m = lm(mixer, d=d)
    a = ids(2, T, 1)
    want = m.forward_carried(a, 64).clone()
    m.forward_carried(a, 64)
    old = [weakref.ref(t) for c in m.held() if c is not None for t in (c if isinstance(c, tuple) else [c]) if torch.is_tensor(t)]
    m.forward_carried(ids(2, 3000, 2), 1024)                          # outgrows every cache
    m.forward_carried(ids(2, 333, 2), 64)
    torch.cuda.synchronize()
    assert all(r() is not None for r in old)
    fill = [torch.full((1 << n,), 1 << 40, device=DEV) for n in range(4, 20) for _ in range(4)]   # whatever was freed is written over
    assert torch.equal(m.forward_carried(a, 64), want)
    del fill


def test_captures_while_another_thread_works():
    """Captures on one thread while another allocates, copies to the host and synchronises its stream: in CUDA's global capture mode
    its first cudaMalloc ends the capture."""
    stop, seen = threading.Event(), []

    def busy():
        n, keep = 0, []
        with torch.cuda.stream(torch.cuda.Stream()):
            while not stop.is_set():
                t = torch.full(((n % 11 + 1) << 20,), 1.0, device=DEV)
                assert float(t[:4].sum()) == 4.0
                torch.cuda.current_stream().synchronize()
                keep = (keep + [t])[-40:]                             # a growing pool: cudaMalloc again and again
                n += 1
        seen.append(n)

    m = lm("aspin")
    want = {T: m.forward_carried(ids(2, T, T), 64).clone() for T in (70, 100, 130, 200)}
    t = threading.Thread(target=busy)
    t.start()
    try:
        for T, w in want.items():
            for _ in range(3):                                        # captured, then replayed
                assert torch.equal(m.forward_carried(ids(2, T, T), 64), w)
        dec = Decoder(m, batch=2)
        dec.prefill(ids(2, 70, 1))
        a = dec.step(ids(2, 1, 2)[:, 0]).clone()
    finally:
        stop.set(); t.join()
    assert seen and seen[0] > 0 and torch.isfinite(a).all()
