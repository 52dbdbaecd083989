"""A layer over a whole sequence of carried windows in one call (mix_windows: the windows side by side for the plain rule, one
rebasing walk for the delta rule) against the same layer called window by window with the state handed on."""
import pytest
import torch
import torch.nn.functional as F

from pragnosia_b200 import _lib, ops, synth
from pragnosia_b200.assoc import AssocCarrier
from pragnosia_b200.model import LM

pytestmark = pytest.mark.gpu
torch.set_grad_enabled(False)
DEV = "cuda"


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize("delta,head_dim", [(False, 64), (True, 64), (True, 128)])
@pytest.mark.parametrize("window,T", [(64, 64), (64, 200), (128, 1), (128, 128), (128, 129), (192, 700), (512, 1333), (1024, 2500)])
@pytest.mark.parametrize("B", [1, 3])
def test_all_windows_at_once_match_window_by_window(delta, head_dim, window, T, B):
    torch.manual_seed(T + window)
    m = AssocCarrier(256, head_dim=head_dim, delta=delta).to(DEV).to(torch.bfloat16)
    m.theta.add_(0.01 * torch.randn_like(m.theta))
    z = torch.randn(B, T, 256, device=DEV).to(torch.bfloat16)
    assert m.windows_fit(window)
    c, H, dk, d = m._consts(), m.h, m.dk, 256
    y = F.linear(z, c["W"], c["b"])                                   # one projection for both: another M may round elsewhere
    outs, S = [], None
    for s in range(0, T, window):
        yw = y[:, s:s + window]
        n = yw.shape[1]
        qkv = [yw[..., i * d:(i + 1) * d].unflatten(-1, (H, dk)) for i in range(3)]
        a, g = yw[..., 3 * d:3 * d + H], yw[..., 3 * d + H:3 * d + 2 * H]
        kw = dict(theta=c["theta"], shift=0.0 if S is None else float(window))
        if delta:
            q, k, v = ops.prep(*qkv, None, c["theta"], torch.arange(n, device=DEV))
            o, S, _ = ops.prefill(q, k, v, m._la(a, c).transpose(1, 2).contiguous(), m._beta(g).transpose(1, 2).contiguous(), S, **kw)
            o = m.on(o).transpose(1, 2).reshape(B, n, d)
        else:
            o, S, _ = ops.layer_prefill(*qkv, g, a, c["A"], m._rot_table(window, c), S, rms_weight=c["onw"], rms_eps=m._rms_eps(), **kw)
        outs.append(o)
    want = F.linear(torch.cat(outs, 1), c["ow"])
    pos = torch.arange(T, device=DEV) % window
    got, S2 = m.mix_windows(z, window, pos, T)
    assert rel(got, want) <= 2e-3 and rel(S2, S) <= 1e-5, (rel(got, want), rel(S2, S))
    tail = (T - 1) % window + 1
    assert rel(m.mix_windows(z, window, pos, tail)[0], got[:, T - tail:]) <= 5e-3


@pytest.mark.parametrize("window,T", [(512, 13 * 512 + 200), (256, 14 * 256 + 1), (1024, 12 * 1024 + 900), (320, 20 * 320)])
def test_windows_of_the_last_round_in_parts(window, T):
    """Twelve chains of more windows than SMs: whole windows, then those of the last round cut into parts (a ragged one last)."""
    test_all_windows_at_once_match_window_by_window(False, 64, window, T, 3)


@pytest.mark.parametrize("window,T", [
    (512, 16 * 512), (512, 16 * 512 - 150), (512, 15 * 512 + 1),      # twelve whole windows a chain, then eight chunks as 3 + 3 + 2; the last one ragged
    (320, 5 * 320 - 30), (320, 17 * 320 + 200), (320, 17 * 320 + 30), # five chunks as 3 + 2, with whole windows ahead of them and without
    (448, 6 * 448), (1024, 3 * 1024 - 70),                            # seven as 4 + 3; sixteen as 4 x 4 with the end inside one
])
def test_windows_in_parts_that_do_not_divide_them(window, T):
    """A part that is shorter than its neighbours ends its window: the first tokens, positions and rotations behind it follow from that."""
    L, B, H = _lib.lib(), 3, 4
    uncut = ((T + window - 1) // window - 1) * B * H * (64 * 64 + 1) * 4
    assert L.pgb_aspin_layer_windows_scratch_bytes(B, H, T, window) > uncut              # more segments than windows: some are cut
    test_all_windows_at_once_match_window_by_window(False, 64, window, T, B)


@pytest.mark.parametrize("n", [4, 5, 16, 17, 128, 129])
def test_combination_of_few_and_many_segments(n):
    """The states entering n later windows: at both sides of the two forms' line, of what is requested ahead and of the factors held at a time."""
    test_all_windows_at_once_match_window_by_window(False, 64, 64, 64 * n + 30, 1)


@pytest.mark.parametrize("mixer", ["aspin", "dspin"])
def test_shape_graphs_and_what_the_caller_keeps(mixer):
    """First call eager, second captured, later ones replayed: the same logits and states every time, and a state kept from one
    call is not overwritten by the next."""
    torch.manual_seed(0)
    m = LM(vocab=256, d=128, layers=2, mlp_mult=2, ctx=64, mixer=mixer, norm="rms").to(DEV).to(torch.bfloat16).eval()
    a, b = (synth.token_ids(2, 150, 256, seed=s).to(DEV) for s in (1, 2))
    la, sa = m.forward_carried(a, return_states=True)
    keep = [s[0].clone() for s in sa]
    m.forward_carried(b)
    for _ in range(2):
        l2, s2 = m.forward_carried(a, return_states=True)
        assert torch.equal(l2, la) and all(torch.equal(x[0], y) for x, y in zip(s2, keep))
        m.forward_carried(b)
        assert all(torch.equal(x[0], y) for x, y in zip(s2, keep))
    assert all(s[1] == 150 % 64 for s in s2)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("T", [1, 31, 33, 100])
def test_prep_with_aligned_rows_matches_the_strided_form(D, T):
    """prep8_kernel (16-byte aligned rows) against prep_kernel (rows offset by four bytes)."""
    B, H = 2, 3
    g = torch.Generator(device=DEV).manual_seed(T)
    buf = torch.randn(3, B, T, H * D + D // 32, device=DEV, generator=g).to(torch.bfloat16)
    views = [b[..., :H * D].unflatten(-1, (H, D)) for b in buf]
    gate = torch.randn(B, T, H, device=DEV, generator=g).to(torch.bfloat16)
    th, pos = synth.rope_theta(H, D).to(DEV), torch.arange(T, device=DEV)
    for x, y in zip(ops.prep(*views, gate, th, pos), ops.prep(*[v.contiguous() for v in views], gate, th, pos)):
        assert (x.float() - y.float()).abs().max() <= 2 ** -7 * x.float().abs().max()


@pytest.mark.parametrize("T", [1, 130, 200])
def test_ragged_windows_by_replay(T):
    """Head dim 128 under the plain rule has no call over all windows: its ragged passes are replayed from the second on."""
    torch.manual_seed(T)
    with torch.device(DEV):
        m = LM(vocab=128, d=256, layers=2, mlp_mult=2, ctx=64, mixer="hspin", norm="rms")
    m = m.to(torch.bfloat16).eval()
    for seed in range(4):
        ids = torch.randint(0, 128, (2, T), device=DEV)
        m.use_graphs = True
        lg, st = m.forward_carried(ids, 64, return_states=True)
        m.use_graphs = False
        want, ws = m.forward_carried(ids, 64, return_states=True)
        assert torch.equal(lg, want) and all(torch.equal(a[0], b[0]) and a[1] == b[1] for a, b in zip(st, ws))


@pytest.mark.parametrize("mixer,d,window", [("aspin", 128, 64), ("dspin", 128, 64), ("hdspin", 256, 128)])
@pytest.mark.parametrize("B,pieces,rest", [(1, 2, 0), (1, 3, 37), (3, 2, 64), (3, 2, 1)])
def test_pieces_of_a_long_sequence(mixer, d, window, B, pieces, rest, monkeypatch):
    """A sequence cut into pieces of whole windows with the states handed on, against the same windows in one piece."""
    from pragnosia_b200 import model as M
    torch.manual_seed(rest)
    m = LM(vocab=256, d=d, layers=2, mlp_mult=2, ctx=window, mixer=mixer, norm="rms").to(DEV).to(torch.bfloat16).eval()
    for mx in m.mix:
        mx.theta.add_(0.01 * torch.randn_like(mx.theta))
    tokens = 2 * window * B
    ids = torch.randint(0, 256, (B, pieces * 2 * window + rest), device=DEV)
    tail = (ids.shape[1] - 1) % window + 1
    (x, y), S = m._layers_windows(ids, window, tail)
    monkeypatch.setattr(M, "WINDOWS_TOKENS", tokens)
    assert m._piece(B, window) == 2 * window
    out = torch.empty_like(torch.stack(S))
    (x1, y1), S1 = m._layers_windows(ids, window, tail, out)
    assert x1.shape == x.shape and all(a.data_ptr() == b.data_ptr() for a, b in zip(S1, out.unbind(0)))
    # bf16 activations of GEMMs with another M: one rounding apart
    assert rel((x1 + y1).float(), (x + y).float()) <= 1e-2 and all(rel(a, b) <= 1e-2 for a, b in zip(S1, S))


def test_a_long_sequence_takes_no_more_memory():
    m = LM(vocab=256, d=768, layers=3, mlp_mult=4, ctx=512, mixer="dspin", norm="rms").to(DEV).to(torch.bfloat16).eval()
    peak = []
    for T in (32768 + 5, 4 * 32768 + 5):
        ids = torch.randint(0, 256, (1, T), device=DEV)
        torch.cuda.synchronize(); torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        m.forward_carried(ids)
        peak.append(torch.cuda.max_memory_allocated() - before)
    assert peak[1] <= 1.05 * peak[0] and peak[1] < 1.5e9, peak


def test_windows_beyond_65535_chunks():
    """The delta rule over a sequence of more chunks than one call of its kernels takes."""
    m = LM(vocab=64, d=64, layers=1, mlp_mult=1, ctx=4096, mixer="dspin", norm="rms").to(DEV).to(torch.bfloat16).eval()
    ids = torch.randint(0, 64, (1, 65536 * 64 + 100), device=DEV)
    lg, S = m.forward_carried(ids, return_states=True)
    # what far-away tokens left has decayed: the end of the sequence alone gives the same
    lg1, S1 = m.forward_carried(ids[:, -(40 * 4096 + 100):], return_states=True)
    assert rel(lg.float(), lg1.float()) < 2e-2 and rel(S[0][0], S1[0][0]) < 2e-2
