"""Captured passes against what changes around them: caches that are outgrown, switches."""
import copy
import threading
import weakref

import pytest
import torch

from pragnosia_b200 import model as M, ops
from pragnosia_b200._lib import lib
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
    old = [weakref.ref(t) for c in m.held() if c is not None for t in c.tensors]
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


@pytest.mark.parametrize("mixer,T", [("aspin", 100), ("dspin", 100), ("aspin", 192), ("hspin", 100)])
@pytest.mark.parametrize("what", ["decoder", "carried"])
def test_two_callers_on_two_streams(mixer, T, what):
    """Two threads, each on a stream of its own, send prompts of one shape through one model, whose captured pass of that shape has
    one set of static tensors: every result is the one its prompt gets alone."""
    m = lm(mixer, d=256, layers=3)
    prompts = [[ids(2, T, 10 * w + i) for i in range(6)] for w in range(2)]

    def run(dec, p):
        if what == "decoder":
            return dec.prefill(p), [st[0] for st in dec.states]
        lg, st = m.forward_carried(p, 64, return_states=True)
        return lg, [s[0] for s in st]

    decs = [Decoder(m, batch=2) for _ in range(2)]
    m.use_graphs = False
    want = [[[t.clone() for t in (r[0], *r[1])] for r in (run(decs[w], p) for p in prompts[w])] for w in range(2)]
    m.use_graphs = True
    for p in (prompts[0][0], prompts[1][0]):
        run(decs[0], p)                                               # seen, then captured
    torch.cuda.synchronize()
    got, start = [[], []], threading.Barrier(2)

    def work(w):
        with torch.no_grad(), torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda._sleep(1000 * (1 + w))
            start.wait()
            for _ in range(10):
                for p in prompts[w]:
                    lg, S = run(decs[w], p)
                    got[w].append([t.clone() for t in (lg, *S)])
            torch.cuda.current_stream().synchronize()

    ts = [threading.Thread(target=work, args=(w,)) for w in range(2)]
    [t.start() for t in ts]; [t.join() for t in ts]
    for w in range(2):
        assert len(got[w]) == 60
        for i, g in enumerate(got[w]):
            assert all(torch.equal(a, b) for a, b in zip(g, want[w][i % 6])), (w, i)


@pytest.mark.parametrize("T", [64, 100])
def test_inside_a_capture_of_the_caller(T):
    m = lm("aspin")
    a = ids(2, T, 1)
    want = m.forward_carried(a, 64).clone()
    m.forward_carried(a, 64)
    g, x = torch.cuda.CUDAGraph(), a.clone()
    with torch.cuda.graph(g):
        out = m.forward_carried(x, 64)
    g.replay()
    assert torch.equal(out, want)


def test_states_of_whole_windows_are_the_callers_own():
    m = lm("aspin", d=1024, layers=2)                                 # 16 heads x 10 sequences: the window graphs
    a, b = ids(10, 128, 1), ids(10, 128, 2)
    _, sa = m.forward_carried(a, 64, return_states=True)
    keep = [s[0].clone() for s in sa]
    m.forward_carried(b, 64)
    assert all(torch.equal(s[0], k) for s, k in zip(sa, keep))


def test_a_copied_model_starts_without_graphs():
    m = lm("aspin")
    a = ids(2, 100, 1)
    want = [m.forward_carried(a, 64) for _ in range(3)][-1]
    c = copy.deepcopy(m)
    assert not c._captured.shapes and torch.equal(c.forward_carried(a, 64), want)


@pytest.mark.parametrize("mixer,d", [("aspin", 256), ("dspin", 256), ("hspin", 256)])
def test_constants_made_on_one_stream_and_used_on_another(mixer, d):
    """The first pass of a model makes the constants its layers cache; a pass on another stream waits for them, and a cache replaced
    meanwhile (another window) is not handed out under that stream's kernels."""
    want = lm(mixer, d=d).forward_carried(ids(2, 100, 1), 64)
    for trial in range(3):
        m = lm(mixer, d=d)
        torch.cuda.synchronize()
        one, two = torch.cuda.Stream(), torch.cuda.Stream()
        with torch.cuda.stream(one):
            torch.cuda._sleep(20_000_000)                             # the constants' kernels are far from done when the other stream starts
            a = m.forward_carried(ids(2, 100, 1), 64)
        with torch.cuda.stream(two):
            b = m.forward_carried(ids(2, 100, 1), 64)
        with torch.cuda.stream(one):
            m.forward_carried(ids(2, 1500, 1), 1024)                  # replaces the tables
            junk = [torch.full((1 << 18,), 7.0, device=DEV) for _ in range(16)]
        torch.cuda.synchronize()
        assert torch.equal(a, want) and torch.equal(b, want)
        del junk


def test_constants_first_made_inside_a_capture_are_not_kept():
    m = lm("aspin", d=256)
    x = torch.randn(2, 70, 256, device=DEV).to(torch.bfloat16)
    layer = m.mix[0]
    want = copy.deepcopy(layer)(x)[0]
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        out = layer(x)[0]
    assert torch.equal(layer(x)[0], want)                             # before the graph has ever run
    g.replay()
    assert torch.equal(out, want)


def test_an_in_place_step_is_not_seen_by_other_callers(monkeypatch):
    """A decode step updates its states where they lie; a layer call from another thread meanwhile leaves the state it was given alone."""
    m = lm("aspin")
    dec = Decoder(m, batch=5, use_graph=False)
    dec.prefill(ids(5, 70, 1))
    z, S = torch.randn(5, 1, 128, device=DEV).to(torch.bfloat16), torch.randn(5, 2, 64, 64, device=DEV)
    keep, step, seen = S.clone(), ops.decode_step, []

    def other():
        with torch.no_grad():
            m.mix[0].mix(z, (S, 3))

    def hook(*a, **k):
        if not seen:
            seen.append(1)
            t = threading.Thread(target=other)
            t.start(); t.join()
        return step(*a, **k)

    monkeypatch.setattr(ops, "decode_step", hook)
    before = dec.states[0][0].clone()
    dec.step(ids(5, 1, 2)[:, 0])
    assert seen and torch.equal(S, keep) and not torch.equal(dec.states[0][0], before)


@pytest.mark.parametrize("mixer", ["aspin", "dspin"])
def test_a_decoder_without_graphs_captures_nothing(mixer):
    m = lm(mixer)
    a = ids(2, 100, 1)
    dec = Decoder(m, batch=2, use_graph=False)
    lg = [dec.prefill(a).clone() for _ in range(4)]
    assert not m._captured.shapes and all(torch.equal(x, lg[0]) for x in lg)
    with_graphs = Decoder(m, batch=2)
    assert all(torch.equal(with_graphs.prefill(a), lg[0]) for _ in range(3)) and any(m._captured.shapes.values())


def test_the_mlps_switch_reaches_the_decode_step(monkeypatch):
    m = lm("aspin")
    calls, linear = [], ops.batch_linear
    monkeypatch.setattr(ops, "batch_linear", lambda *a, **k: calls.append(k.get("act")) or linear(*a, **k))
    dec = Decoder(m, batch=6, use_graph=False)
    out = []
    for fused in (True, False):
        for mp in m.mlp:
            mp.fused_up = fused
        dec.prefill(ids(6, 70, 1))
        calls.clear()
        out.append(dec.step(ids(6, 1, 2)[:, 0]).float())
        assert calls.count("gelu") == (len(m.mlp) if fused else 0)
    assert float((out[0] - out[1]).norm() / out[1].norm()) < 2e-2


@pytest.mark.parametrize("B,T,window", [(1, 64, 64), (2, 200, 64), (2, 257, 128)])
def test_the_single_role_variant_reaches_windows(B, T, window):
    """pgb_tc_set_variant(1): a pass over windows is that kernel window by window, and a graph captured before is retired."""
    L = lib()
    m = lm("aspin", d=256)
    a = ids(B, T, 1)
    first = [m.forward_carried(a, window) for _ in range(3)][-1]
    layer = m.mix[0]
    z, S0 = torch.randn(B, T, 256, device=DEV).to(torch.bfloat16), torch.randn(B, 4, 64, 64, device=DEV)
    c = layer._consts()
    y = torch.nn.functional.linear(z, c["W"], c["b"])
    try:
        assert L.pgb_tc_set_variant(1) == 0 and L.pgb_variants() == 1
        S, outs = S0, []
        for s in range(0, T, window):
            yw = y[:, s:s + window]
            q, k, v = (yw[..., i * 256:(i + 1) * 256].unflatten(-1, (4, 64)) for i in range(3))
            o, S, _ = ops.layer_prefill(q, k, v, yw[..., 772:776], yw[..., 768:772], c["A"], layer._rot_table(window, c), S, theta=c["theta"],
                                        shift=float(window), rms_weight=c["onw"], rms_eps=layer._rms_eps())
            outs.append(o)
        q, k, v = (y[..., i * 256:(i + 1) * 256].unflatten(-1, (4, 64)) for i in range(3))
        o, S1 = ops.layer_prefill_windows(q, k, v, y[..., 772:776], y[..., 768:772], c["A"], layer._rot_table(window, c), c["theta"], window, c["onw"],
                                          layer._rms_eps(), S0=S0)
        assert torch.equal(o, torch.cat(outs, 1)) and torch.equal(S1, S)
        second = m.forward_carried(a, window)
        assert L.pgb_variants() == m._captured.stamp[1] == 1
    finally:
        L.pgb_tc_set_variant(0)
    assert float((first.float() - second.float()).norm() / first.float().norm()) < 2e-2


@pytest.mark.parametrize("sms,over_all", [(3, False), (4, False), (5, True)])
def test_the_form_of_a_pass_follows_the_devices_sm_count(sms, over_all, monkeypatch):
    """Four chains of two sequences: one call over all windows where there are more SMs than that, else the graph window by window."""
    m = lm("aspin")
    a = ids(2, 128, 1)
    want = m.forward_carried(a, 64)
    monkeypatch.setattr(M, "sm_count", lambda device: sms)
    m._captured.windows.clear()
    got = m.forward_carried(a, 64)
    assert bool(m._captured.windows) != over_all
    assert float((got.float() - want.float()).norm() / want.float().norm()) < 2e-2


@pytest.mark.parametrize("mixer", ["aspin", "dspin"])
def test_no_room_for_a_captured_pass(mixer):
    """Memory for an eager pass but not for a graph's own copy of its activations: the pass runs eagerly."""
    m = lm(mixer, d=512, layers=2)
    a = ids(4, 4000, 1)
    want = m.forward_carried(a, 64).clone()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    m._captured.shapes.clear()
    m.forward_carried(a, 64)                                          # eagerly: what it takes
    torch.cuda.synchronize()
    total, peak = torch.cuda.get_device_properties(0).total_memory, torch.cuda.max_memory_reserved()
    torch.cuda.set_per_process_memory_fraction((peak + (4 << 20)) / total)
    try:
        out = [m.forward_carried(a, 64) for _ in range(3)]
        assert list(m._captured.shapes.values()) == [M._NO_ROOM]
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert all(torch.equal(x, want) for x in out)
    m._captured.shapes.clear()
    out = [m.forward_carried(a, 64) for _ in range(3)]
    assert all(m._captured.shapes.values()) and all(torch.equal(x, want) for x in out)


def test_constants_nobody_has_marked_yet():
    """Made by a call that has not come to its end (here: the constants alone); the other stream marks their stream itself."""
    want = lm("aspin", d=256).mix[0]
    x = torch.randn(2, 70, 256, device=DEV).to(torch.bfloat16)
    want = want(x)[0]
    layer = lm("aspin", d=256).mix[0]
    torch.cuda.synchronize()
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(one):
        torch.cuda._sleep(20_000_000)
        layer._consts()
        assert layer._fused.mark.due
    with torch.cuda.stream(two):
        got = layer(x)[0]
    assert not layer._fused.mark.due
    torch.cuda.synchronize()
    assert torch.equal(got, want)


@pytest.mark.parametrize("name", ["a", "b"])
def test_replaced_mlp_layers_are_called(name):
    """A layer of the MLP that is more than its weight (an adapter, say) keeps its own forward in the decode step of a batch."""
    class Adapted(torch.nn.Linear):
        def forward(self, x):
            return super().forward(x) * 3

    m = lm("aspin")
    dec = Decoder(m, batch=6, use_graph=False)
    dec.prefill(ids(6, 70, 1))
    plain = dec.step(ids(6, 1, 2)[:, 0]).float()
    for mp in m.mlp:
        old = getattr(mp, name)
        new = Adapted(old.in_features, old.out_features).to(DEV).to(torch.bfloat16)
        new.load_state_dict(old.state_dict())
        setattr(mp, name, new)
    dec.prefill(ids(6, 70, 1))
    got = dec.step(ids(6, 1, 2)[:, 0]).float()
    for mp in m.mlp:                                                  # the same as weights
        lin = getattr(mp, name)
        setattr(mp, name, torch.nn.Linear(lin.in_features, lin.out_features).to(DEV).to(torch.bfloat16))
        getattr(mp, name).load_state_dict({k: 3 * v for k, v in lin.state_dict().items()})
    dec.prefill(ids(6, 70, 1))
    want = dec.step(ids(6, 1, 2)[:, 0]).float()
    assert float((got - want).norm() / want.norm()) < 2e-2 < float((plain - want).norm() / want.norm())


def test_the_benchmarks_decode_leg_times_no_capture(monkeypatch):
    """Both timed calls of a leg, the sampled loop and the prompt pass subtracted from it, replay what is captured by then."""
    import types
    import bench
    from pragnosia_b200 import kernel_bench
    model = LM(vocab=bench.CFG["vocab"], d=128, layers=2, mlp_mult=4, ctx=512, mixer="aspin", norm="rms").cuda().bfloat16().eval()
    captures, calls, capture, generate, prefill = [0], [], LM.capture, Decoder.generate, Decoder.prefill

    def counted(*a, **k):
        captures[0] += 1
        return capture(*a, **k)

    def logged(name, f):
        def call(*a, **k):
            before, out = captures[0], f(*a, **k)
            calls.append((name, captures[0] - before))
            return out
        return call

    monkeypatch.setattr(LM, "capture", counted)
    monkeypatch.setattr(Decoder, "generate", logged("generate", generate))
    monkeypatch.setattr(Decoder, "prefill", logged("prefill", prefill))
    monkeypatch.setattr(kernel_bench, "time_case", lambda name: (1.0, 1.0))
    bench.decode_numbers(model, torch.device("cuda"), dict(hbm_gbs=1.0), types.SimpleNamespace(decode_steps=8))
    timed = [i for i, (name, _) in enumerate(calls) if name == "generate"][1::2]      # per batch: the warm-up, then the timed call
    assert len(timed) == 2 and sum(n for _, n in calls) >= 4                          # per batch, the prompt and the token
    for i in timed:
        assert calls[i] == ("generate", 0) and calls[i + 1] == ("prefill", 0), calls
