"""The language model around the carrier layers: same constructor arguments, parameter names and carried-state
interface as the reference's src/model.py LM (:621-864), restricted to the pure-carrier mixers (aspin, dspin, hspin,
hdspin, fspin). Attention controls, hybrids, growth and the training loss are other subsystems and are not here."""
from __future__ import annotations

import contextlib
import threading

import torch
import torch.nn as nn
import torch.nn.functional as F

from . import ops
from ._lib import Cached, graph_capture, lib, mark_constants, sm_count, warm_up
from .assoc import AssocCarrier
from .spin import SpinCarrier


class MLP(nn.Module):
    """norm -> Linear(mult*d) -> GELU -> Linear(d), residual (src/model.py:552-560)."""

    def __init__(self, d: int, mult: int = 4):
        super().__init__()
        self.n = nn.LayerNorm(d)
        self.a = nn.Linear(d, mult * d)
        self.b = nn.Linear(mult * d, d)

    def forward(self, x):
        return x + self.ff(self.n(x))

    fused_up = True     # bf16 on CUDA: Linear(d, mult*d) + GELU as one tensor-core GEMM with the activation in its epilogue

    def ff(self, z):
        """The block without its norm and residual add."""
        if (self.fused_up and type(self.a) is nn.Linear and z.is_cuda and z.dtype == torch.bfloat16 and self.a.weight.dtype == torch.bfloat16
                and z.shape[-1] % 8 == 0 and self.a.weight.shape[0] % 8 == 0 and z.numel() // z.shape[-1] >= 128):
            return self.b(ops.linear_act(z, self.a.weight, self.a.bias, act="gelu"))
        return self.b(F.gelu(self.a(z)))


_MIXERS = {
    "aspin": lambda d: AssocCarrier(d), "dspin": lambda d: AssocCarrier(d, delta=True),
    "hspin": lambda d: AssocCarrier(d, head_dim=128), "hdspin": lambda d: AssocCarrier(d, delta=True, head_dim=128),
    "fspin": lambda d: SpinCarrier(d, gated="rf"),
}


# Tokens of a batch that one pass over many windows takes at most: activations of 12 KB a token at width 768 (20 under the delta
# rule: 0.63 GB in all), and GEMMs that long gain nothing from more rows.
WINDOWS_TOKENS = 32768


class LM(nn.Module):
    def __init__(self, vocab=8192, d=768, layers=12, mlp_mult=4, ctx=512, mixer="aspin", norm="ln"):
        super().__init__()
        if mixer not in _MIXERS:
            raise NotImplementedError(f"mixer {mixer!r}: only the pure-carrier mixers {sorted(_MIXERS)} are built here")
        self.vocab, self.d, self.layers, self.ctx, self.mixer, self.norm = vocab, d, layers, ctx, mixer, norm
        self.wavefront = True                                # graphed forward_carried: consecutive windows a layer apart on separate streams
        self.wavefront_streams = 4
        self.e = nn.Embedding(vocab, d)
        self.p = nn.Embedding(ctx, d)
        self.mix = nn.ModuleList([_MIXERS[mixer](d) for _ in range(layers)])
        self.mlp = nn.ModuleList([MLP(d, mlp_mult) for _ in range(layers)])
        self.n = nn.LayerNorm(d)
        self.use_graphs = True          # CUDA: replay one captured graph per window in forward_carried
        self._captured = _Captured()
        self._wpos = None
        if norm == "rms":                      # every residual-stream LayerNorm becomes an RMSNorm of the same width
            for mod in list(self.modules()):
                for nm, child in list(mod.named_children()):
                    if isinstance(child, nn.LayerNorm):
                        setattr(mod, nm, nn.RMSNorm(child.normalized_shape[0]))
        self.apply(self._init)

    @staticmethod
    def _init(m):
        if isinstance(m, (nn.Embedding, nn.Linear)):
            nn.init.normal_(m.weight, 0.0, 0.02)
            if getattr(m, "bias", None) is not None:
                nn.init.zeros_(m.bias)

    def weights_stamp(self):
        """Changes whenever a captured graph of this model would compute with something stale: a parameter that moved
        (another dtype or device), a mixer whose derived constants must be rebuilt (an in-place update, load_state_dict), or
        another kernel variant chosen (pgb_tc_set_variant and its like)."""
        ptrs = tuple(p.data_ptr() for p in self.parameters())
        return ptrs, lib().pgb_variants(), tuple(mx.consts_key() for mx in self.mix if isinstance(mx, AssocCarrier))

    def _embed(self, x):
        return self.e(x) + self.p(torch.arange(x.shape[1], device=x.device) % self.p.num_embeddings)

    @staticmethod
    def _add_norm(x, delta, norm):
        """y = x + delta, z = norm(y) in one kernel where the row length allows it; else the two torch ops."""
        d = x.shape[-1]
        lim = (2048, 8) if x.dtype == torch.bfloat16 else (1024, 4)
        if x.dtype in (torch.bfloat16, torch.float32) and d <= lim[0] and d % lim[1] == 0 and not torch.is_grad_enabled():
            return ops.add_norm(x, delta, norm)
        y = x if delta is None else x + delta
        return y, norm(y)

    def _layers(self, h, states, inplace=None):
        """Every (mixer, MLP) pair over h. Returns (x, delta): the residual stream and the last block's not-yet-added
        output, so the caller's final norm fuses that add as well. Each block's input norm is fused with the previous
        block's residual add. inplace: the associative layers update the states where they lie (None: as each layer is set)."""
        x, delta = h, None
        for i, (mx, mp) in enumerate(zip(self.mix, self.mlp)):
            x, z = self._add_norm(x, delta, mx.ln)
            delta, states[i] = mx.mix(z, states[i], inplace) if isinstance(mx, AssocCarrier) else mx.mix(z, states[i])
            x, z = self._add_norm(x, delta, mp.n)
            delta = mp.ff(z)
        return x, delta

    def windows_fit(self, window: int) -> bool:
        return (self.e.weight.is_cuda and self.e.weight.dtype == torch.bfloat16 and
                all(isinstance(mx, AssocCarrier) and mx.windows_fit(window) for mx in self.mix))

    def held(self):
        """What the kernels of a pass read beside the parameters: constants the mixers and this model derive and cache. Each cache
        is replaced when it is outgrown (a longer window, another sequence length), so a captured graph keeps these itself."""
        return [getattr(mx, n, None) for mx in self.mix for n in ("_fused", "_rot", "_pos")] + [self._wpos]

    def capture(self, stream, run, pool=None):
        """(graph of run(), what run returned, what the graph reads and must keep). Behind a warm_up() on the same stream."""
        while True:
            held, graph = self.held(), torch.cuda.CUDAGraph()
            with graph_capture(graph, stream, pool):
                out = run()
            if all(a is b for a, b in zip(held, self.held())):        # else another thread replaced a cache meanwhile: once more
                return graph, out, held

    def _window_positions(self, T, window, device):
        """(position inside its window of every token, the same modulo the position table) for the first T tokens."""
        got = self._wpos
        both = got.get() if got is not None and got.key == (window, device) and got.value[0].numel() >= T else None
        if both is None:
            pos = torch.arange(T, device=device) % window
            both = (pos, pos % self.p.num_embeddings)
            self._wpos = Cached((window, device), both, both).keep(got)
        return tuple(t[:T] for t in both)

    def _piece(self, B, window):
        """Tokens of a sequence that go through the layers together: whole windows, WINDOWS_TOKENS tokens over the batch at most (or
        one window)."""
        return window * max(1, WINDOWS_TOKENS // (B * window))

    def _layers_windows(self, ids, window, tail, states=None):
        """Every layer over many windows of the sequence at once: layer l of a window needs the layer below on that window
        and, of the window before, only this layer's state, so nothing but the carried state inside a layer is sequential --
        one set of GEMMs per layer over all of them instead of one per window. A sequence longer than a piece goes through piece by
        piece with the states handed on, so the activations' memory does not grow with it. Returns (x, delta) of the last `tail`
        tokens (the last layer is computed for those only behind its scan) and the layers' final states, written into
        `states` (tensors) when given."""
        B, T = ids.shape
        piece, last, S = self._piece(B, window), self.layers - 1, [None] * self.layers
        for s in range(0, T, piece):
            n, end = min(piece, T - s), s + piece >= T
            wpos, epos = self._window_positions(n, window, ids.device)
            x, delta, new = self.e(ids[:, s:s + n]) + self.p(epos), None, []
            for i, (mx, mp) in enumerate(zip(self.mix, self.mlp)):
                x, z = self._add_norm(x, delta, mx.ln)
                keep = n if i != last else tail if end else 0
                delta, Si = mx.mix_windows(z, window, wpos, keep, states[i] if end and states is not None else None, S[i])
                new.append(Si)
                if keep == 0:
                    break
                x, z = self._add_norm(x if keep == n else x[:, n - keep:], delta, mp.n)
                delta = mp.ff(z)
            S = new
        return (x, delta), S

    def _by_window(self, ids, window, tail, states=None):
        """What _layers_windows returns, window by window (mixers without a call over all of them)."""
        new = [None] * self.layers
        for s in range(0, ids.shape[1], window):
            last = self._layers(self._embed(ids[:, s:s + window]), new)
        S = [st[0] for st in new]
        if states is not None:
            torch._foreach_copy_(list(states), S)
            S = states
        return last, S

    def _replays(self, window: int) -> bool:
        """Whether a pass window by window is the same kernels on the same addresses every time: no option in the way."""
        return (self.use_graphs and self.e.weight.is_cuda and self.e.weight.dtype == torch.bfloat16 and
                all(isinstance(mx, AssocCarrier) and mx.plain_step and mx.pos_wrap is None and not mx.need_sent for mx in self.mix))

    def _windows_pass(self, ids, window, tail, graphs=True):
        """_layers_windows (or _by_window where that does not fit) and the final norm, from the second call with a shape on as one
        CUDA-graph replay (the first call of a shape runs eagerly: a shape that never comes back is not worth a capture; nor is a pass
        of several pieces, whose kernels take longer than their launches). Returns (z (B,tail,d), states), both the caller's own.
        graphs=False, or a caller that is capturing: eagerly."""
        body = self._layers_windows if self.windows_fit(window) else self._by_window
        if graphs and self._may_replay(ids) and ids.shape[1] <= self._piece(ids.shape[0], window):
            with self._captured.turn(self) as c:
                run = c.shape_graph(self, ids, body, window, tail)
                if run is not None:
                    last, states = run(ids)
                    return self._add_norm(*last, self.n)[1], states
        last, states = body(ids, window, tail)
        if ids.is_cuda:
            mark_constants(ids)
        return self._add_norm(*last, self.n)[1], states

    def _may_replay(self, ids) -> bool:
        return self.use_graphs and ids.is_cuda and not torch.cuda.is_current_stream_capturing()

    def trunk(self, x, states=None, carry=False):
        """Everything but the output head; with carry=True also takes / returns the per-layer states."""
        new = list(states) if states is not None else [None] * self.layers
        h = self._add_norm(*self._layers(self._embed(x), new), self.n)[1]
        return (h, new) if carry else h

    def forward(self, x, return_hidden=False):
        h = self.trunk(x)
        logits = F.linear(h, self.e.weight)
        return (logits, h) if return_hidden else logits

    @torch.no_grad()
    def forward_carried(self, x, window=None, return_states=False):
        """A sequence longer than ctx, window by window with the carrier state carried; logits of the FINAL window only
        (src/model.py:843-864). The head runs once, on the last window (the reference computes and discards it for every
        window). On CUDA, with use_graphs set and whole windows, each window pass is one CUDA-graph replay."""
        window = window or self.ctx
        B, T = x.shape
        tail = (T - 1) % window + 1
        # Fewer chains than SMs, or a ragged last window: layer by layer over the whole sequence (or, on mixers without a call over all
        # windows, window by window: seven launches a layer and window, whose issue from Python took longer than they did). With more
        # chains and whole windows the window-by-window graph below keeps the GPU as full and its activations in the L2.
        all_windows = self.windows_fit(window) and x.is_cuda and (B * self.mix[0].h < sm_count(x.device) or T % window)
        whole = T % window == 0 and T >= window
        if all_windows or (x.is_cuda and self._replays(window) and not whole):
            z, states = self._windows_pass(x, window, tail)
            states = [(S, tail) for S in states]
        elif whole and self._may_replay(x):
            with self._captured.turn(self) as c:
                last, states = c.window_graphs(self, x, window)
                z = self._add_norm(*last, self.n)[1]
                if return_states:                                     # the graph's own are overwritten by the next call
                    own = [t for st in states for t in st if torch.is_tensor(t)]
                    kept = [torch.empty_like(t) for t in own]
                    torch._foreach_copy_(kept, own)
                    it = iter(kept)
                    states = [tuple(next(it) if torch.is_tensor(t) else t for t in st) for st in states]
        else:
            states = [None] * self.layers
            last = None
            for s in range(0, T, window):
                last = self._layers(self._embed(x[:, s:s + window]), states)
            z = self._add_norm(*last, self.n)[1]
        logits = F.linear(z, self.e.weight)
        return (logits, states) if return_states else logits


_NO_ROOM = "no room"                    # in place of a captured pass whose memory could not be had: eagerly from then on


class _Captured:
    """A model's captured passes. They write static tensors of their own and share one memory pool, so they run one at a time:
    turn() holds the host lock, makes the current stream wait for the turn before (whichever thread and stream it came from) and
    drops every graph once the weights' stamp has changed. Results are copied out before a turn ends. A copy or a pickle of the
    model starts with none."""

    def __init__(self):
        self.lock, self.done = threading.RLock(), None
        self.stamp = self.pool = self.stream = None
        self.windows = {}               # whole windows: (batch, window, windows) -> _StepGraph, (batch, window) -> _WindowGraphs
        self.shapes = {}                # passes over many windows: shapes seen (False) and captured, in order of use

    def __deepcopy__(self, memo):
        return type(self)()

    def __reduce__(self):
        return type(self), ()

    @contextlib.contextmanager
    def turn(self, model):
        with self.lock:
            here = torch.cuda.current_stream()
            if self.done is None:
                self.done = torch.cuda.Event()
            else:
                here.wait_event(self.done)
            # A captured graph holds the addresses of the parameters and of the constants the mixers derive from them
            # (the concatenated projection weight, the gated output weight): any change of either retires every graph.
            stamp = model.weights_stamp()
            if stamp != self.stamp:
                self.windows.clear()
                self.shapes.clear()
                self.stamp, self.pool = stamp, None
            try:
                yield self
            finally:
                self.done.record(here)

    def shape_graph(self, model, ids, body, window, tail):
        """The captured pass of this shape; None the first time it comes, and where there is no room for it."""
        key = (tuple(ids.shape), ids.dtype, window, tail, ids.device)
        run = self.shapes.pop(key, None)
        if run is _NO_ROOM:
            self.shapes[key] = run
            return None
        if run is None:
            self.shapes[key] = False
            if len(self.shapes) > 64:
                self.shapes.pop(next(iter(self.shapes)))
            return None
        if run is False:
            held = [k for k, v in self.shapes.items() if isinstance(v, _ShapeGraph)]
            if len(held) >= 8:                                        # eight captured shapes at most, the longest unused one goes
                self.shapes.pop(held[0])
            if self.pool is None:
                self.pool, self.stream = torch.cuda.graph_pool_handle(), torch.cuda.Stream()
            try:
                run = _ShapeGraph(model, ids, body, window, tail, self.stream, self.pool)
            except torch.cuda.OutOfMemoryError:                       # no room for a second set of activations: give back what is held
                self.shapes.clear()
                self.shapes[key], self.pool = _NO_ROOM, None
                return None
        self.shapes[key] = run                                        # last in the order: most recently used
        return run

    def window_graphs(self, model, x, window):
        """((x, delta) of the last window, states) of a pass over whole windows."""
        B, T = x.shape
        nw = T // window
        if model.wavefront and nw >= 2 and all(isinstance(mx, AssocCarrier) for mx in model.mix):
            # every window of the call in ONE graph, consecutive windows on two streams a layer apart
            key = (B, window, nw, x.device, model.e.weight.dtype)
            run = self.windows.get(key)
            if run is None:
                run = self.windows[key] = _StepGraph(model, B, window, nw, x.device)
            last = run(x)
        else:
            key = (B, window, x.device, model.e.weight.dtype)
            run = self.windows.get(key)
            if run is None:
                run = self.windows[key] = _WindowGraphs(model, B, window, x.device)
            for s in range(0, T, window):
                last = run(x[:, s:s + window], first=(s == 0))
        return last, run.states


class _ShapeGraph:
    """One captured _layers_windows or _by_window: static ids in, (x, delta) of the last tokens and one tensor of every layer's final state
    out (cloned per call, so that what a caller keeps is not overwritten by the next one). All of them lie in the graph's pool."""

    def __init__(self, model, ids, body, window, tail, stream, pool):
        mx = model.mix[0]

        def run():
            self.ids = torch.empty_like(ids)
            self.states = torch.empty(model.layers, ids.shape[0], mx.h, mx.dk, mx.dk, device=ids.device, dtype=torch.float32)
            return body(self.ids, window, tail, self.states)[0]

        with warm_up(stream):
            body(ids, window, tail)
            self.graph, self.out, self.held = model.capture(stream, run, pool)

    def __call__(self, ids):
        self.ids.copy_(ids)
        self.graph.replay()
        return self.out, list(self.states.clone().unbind(0))


class _StepGraph:
    """ONE CUDA graph of a whole multi-window pass, with consecutive windows on separate streams. Window w + 1 needs from
    window w only each layer's carried state, so it can run one layer behind it instead of after it: layer l of window
    w + 1 waits for the event recorded after layer l of window w. The two windows' kernels then share the GPU -- the
    half-empty second wave of one window's prefill kernel (192 one-per-SM CTAs on 148 SMs) is filled by the other
    window's GEMM tiles. Same kernels in the same order along every dependency chain: results are those of the
    window-by-window pass to the bit. The reference runs the windows one after the other, eagerly (src/model.py:857-863)."""

    def __init__(self, model, B, Tw, NW, device):
        self.m, self.B, self.Tw, self.NW = model, B, Tw, NW
        self.ids = torch.zeros(B, Tw * NW, dtype=torch.long, device=device)
        self.sides = [torch.cuda.Stream(device=device) for _ in range(min(NW, model.wavefront_streams) - 1)]
        self.graph = None
        self.states = None
        self.out = None

    def _pass(self):
        m, main = self.m, torch.cuda.current_stream()
        streams = [main] + self.sides
        states = [None] * m.layers
        fork = torch.cuda.Event(); fork.record(main)
        for sd in self.sides:
            sd.wait_event(fork)
        prev, out = None, None
        for w in range(self.NW):
            st = streams[w % len(streams)]
            evs = [torch.cuda.Event() for _ in range(m.layers)]
            with torch.cuda.stream(st):
                x, delta = m._embed(self.ids[:, w * self.Tw:(w + 1) * self.Tw]), None
                for i, (mx, mp) in enumerate(zip(m.mix, m.mlp)):
                    x, z = m._add_norm(x, delta, mx.ln)
                    if prev is not None:
                        st.wait_event(prev[i])                         # the state this layer enters with
                    delta, states[i] = mx.mix(z, states[i], inplace=w > 0)     # later windows update the first window's state tensors
                    evs[i].record(st)
                    x, z = m._add_norm(x, delta, mp.n)
                    delta = mp.ff(z)
                out = (x, delta)
            prev = evs
        for sd in self.sides:
            join = torch.cuda.Event(); join.record(sd); main.wait_event(join)
        return out, states

    def __call__(self, ids):
        if self.graph is None:
            main = torch.cuda.Stream()
            with warm_up(main):
                self._pass()
                main.synchronize()                                     # the pass's tensors crossed streams; they are free from here on
                self.graph, (self.out, self.states), self.held = self.m.capture(main, self._pass)
        self.ids.record_stream(torch.cuda.current_stream())            # made on the first caller's stream
        self.ids.copy_(ids)
        self.graph.replay()
        return self.out


class _WindowGraphs:
    """Two CUDA graphs of one window pass (embedding and every layer over a static (B,Tw) block of ids): one for a
    sequence's first window (no entering state) and one for every later window, which updates the per-layer state
    buffers in place. The reference runs this loop eagerly (src/model.py:857-863); at small batch it is launch-bound."""

    def __init__(self, model, B, Tw, device):
        self.m, self.B, self.Tw = model, B, Tw
        self.ids = torch.zeros(B, Tw, dtype=torch.long, device=device)
        self.states = None
        self.first = self.later = None
        self.out_first = self.out_later = None

    def _pass(self, states, inplace):
        m = self.m
        new = list(states)
        out = m._layers(m._embed(self.ids), new, inplace)
        if inplace:                            # states that came back as new tensors (the diagonal carrier) are copied home
            for old, cur in zip(states, new):
                for a, b in zip(old, cur):
                    if torch.is_tensor(a) and a.data_ptr() != b.data_ptr():
                        a.copy_(b)
        return out, new

    def _capture(self):
        none = [None] * self.m.layers
        side = torch.cuda.Stream()
        with warm_up(side):
            _, st = self._pass(none, False)
            self._pass(st, True)
            self.first, (self.out_first, self.states), held = self.m.capture(side, lambda: self._pass(none, False))
            self.later, (self.out_later, _), held2 = self.m.capture(side, lambda: self._pass(self.states, True), self.first.pool())
            self.held = held + held2

    def __call__(self, ids, first):
        if self.first is None:
            self._capture()
        self.ids.record_stream(torch.cuda.current_stream())            # made on the first caller's stream
        self.ids.copy_(ids)
        if first:
            self.first.replay()
            return self.out_first
        self.later.replay()
        return self.out_later
