"""The decode step as ONE launch per token (decode_flow.cu; decode_token.cu, with barriers, where it is asked for) against the same step
chained from this library's separate kernels (five launches a layer), whose parity with the oracle the model tests pin: same roundings,
sums of the same fp32 products in an order that the row length decides, so logits and states are compared at a few bf16 ulps. Ids are
exact between graph and eager launches of one step."""
import pytest
import torch

from pragnosia_b200 import _lib, synth
from pragnosia_b200.generate import Decoder

from test_gpu_model import DEV, close, small_lm

pytestmark = pytest.mark.gpu


def healthy():
    import ctypes
    flag = ctypes.c_int(-1)
    assert _lib.lib().pgb_tc_error_flag(ctypes.byref(flag)) == 0
    return flag.value


@pytest.mark.parametrize("mixer,norm", [("aspin", "rms"), ("aspin", "ln"), ("dspin", "ln"), ("hspin", "rms"), ("hdspin", "ln")])
@pytest.mark.parametrize("B", [1, 2, 3, 4])
def test_one_launch_step_matches_the_chained_kernels(mixer, norm, B):
    m, _, _ = small_lm(mixer, norm, torch.bfloat16)
    ids = synth.token_ids(B, 60, 256, seed=23).to(DEV)
    outs = {}
    for token_kernel in (False, True):
        for use_graph in (False, True):
            dec = Decoder(m, batch=B, use_graph=use_graph, token_kernel=token_kernel)
            assert dec._fused_ok() and dec._token_ok() == token_kernel
            assert dec.launches_per_token == (2 if token_kernel else 3 + 5 * m.layers)
            lg = [dec.prefill(ids[:, :40])]
            for t in range(40, 60):                                   # crosses the window edge (ctx 32): the position wraps
                lg.append(dec.step(ids[:, t]).clone())
            outs[(token_kernel, use_graph)] = (torch.stack(lg, 1), [st[0].clone() for st in dec.states])
    ref_lg, ref_S = outs[(False, False)]
    for key, (lg, S) in outs.items():
        close(lg, ref_lg, 2e-2, f"logits one-launch={key[0]} graph={key[1]}")
        for a, b in zip(S, ref_S):
            close(a, b, 5e-3, f"state one-launch={key[0]} graph={key[1]}")
    # rows this short are summed in the chained kernels' order: most logits agree to the bit
    same = (outs[(True, True)][0] == ref_lg).float().mean().item()
    assert same > 0.9, same
    assert healthy() == 0


def test_generate_through_the_one_launch_step():
    m, _, _ = small_lm("aspin", "ln", torch.bfloat16)
    prompt = synth.token_ids(2, 40, 256, seed=3).to(DEV)
    for temp in (0.0, 1.0):
        a = Decoder(m, batch=2).generate(prompt, 24, temp=temp, seed=5)
        b = Decoder(m, batch=2, token_kernel=False).generate(prompt, 24, temp=temp, seed=5)
        c = Decoder(m, batch=2, use_graph=False).generate(prompt, 24, temp=temp, seed=5)
        assert tuple(a.shape) == (2, 24)
        assert torch.equal(a, c)                                      # graph replay and eager launches draw the same ids
        assert (a == b).float().mean().item() > 0.9                   # and the chained kernels' ids
    d = Decoder(m, batch=2)
    first = d.generate(prompt, 8, temp=0.0)
    again = d.generate(prompt, 8, temp=0.0)                           # the decoder, its table and its counters are reusable
    assert torch.equal(first, again)
    assert healthy() == 0


def test_changed_weights_retire_the_table():
    m, _, _ = small_lm("aspin", "rms", torch.bfloat16)
    prompt = synth.token_ids(1, 40, 256, seed=4).to(DEV)
    d = Decoder(m, batch=1)
    d.prefill(prompt); lg0 = d.step(prompt[:, -1]).clone()
    with torch.no_grad():
        m.mix[0].o.weight.mul_(0.5)                                   # the folded output weight is rebuilt, at a new address
    d.prefill(prompt); lg1 = d.step(prompt[:, -1]).clone()
    ref = Decoder(m, batch=1, token_kernel=False); ref.prefill(prompt)
    close(lg1, ref.step(prompt[:, -1]), 2e-2, "after the update")
    assert not torch.equal(lg0, lg1)


@pytest.mark.parametrize("d,mixer,mult,vocab,norm", [
    (64, "aspin", 1, 40, "rms"),                                       # fewer rows than CTAs
    (192, "dspin", 12, 300, "ln"),                                     # MLP down with its rows shared across the warps (K 2304)
    (256, "hspin", 9, 9600, "ln"),                                     # the same on a multiple of eight warps only; a head of several rounds
    (1280, "hdspin", 4, 5000, "rms"),                                  # phases of several rounds, rows too long for four a warp
])
@pytest.mark.parametrize("B", [1, 3])
def test_step_without_barriers_matches_the_one_with(d, mixer, mult, vocab, norm, B, monkeypatch):
    """Same roundings, and but for rows shared across warps (fp32 sums in another order: a bf16 rounding may fall the other way, 2^-8) the
    same order of every sum."""
    from pragnosia_b200 import ops
    from pragnosia_b200.model import LM
    torch.manual_seed(d)
    m = LM(vocab=vocab, d=d, layers=3, mlp_mult=mult, ctx=16, mixer=mixer, norm=norm).to(DEV).bfloat16().eval()
    ids = synth.token_ids(B, 40, vocab, seed=d).to(DEV)
    outs = []
    for flow in (True, False):
        if not flow:
            monkeypatch.setattr(ops, "decode_flow_work_bytes", lambda *a: 0)
        dec = Decoder(m, batch=B)
        lg = [dec.prefill(ids[:, :20])]
        for t in range(20, 30):                                       # crosses the window's edge (ctx 16)
            lg.append(dec.step(ids[:, t]).clone())
        lg.append(dec.prefill(ids[:, :17]))                           # a new prompt on the same decoder: the words keep their marks
        lg.append(dec.step(ids[:, 17]).clone())
        assert dec._plan["flow"] == flow
        outs.append((torch.stack(lg, 1), [st[0].clone() for st in dec.states]))
    close(outs[0][0], outs[1][0], 2e-2, "logits")
    for a, b in zip(outs[0][1], outs[1][1]):
        close(a, b, 5e-3, "state")
    if mult * d < 2048 or d > 1000:
        assert (outs[0][0] == outs[1][0]).float().mean().item() > 0.9
    assert healthy() == 0


def test_a_barrier_wait_that_runs_out_raises_the_flag_and_returns():
    """The grid barrier's failure path without a fault: one CTA waits, with a short limit, for arrivals that never come."""
    import ctypes
    assert healthy() == 0
    sync = torch.zeros(2, dtype=torch.int64, device=DEV)
    rc = _lib.lib().pgb_decode_token_wait_selftest(ctypes.c_void_p(sync.data_ptr()), 2000, None)
    assert rc == 0
    torch.cuda.synchronize()
    assert sync.tolist() == [1, 1]                                    # it did arrive, and gave up
    assert healthy() == 81 and healthy() == 0                         # reported once, then clear
    x = torch.ones(8, device=DEV)                                     # the context is still usable
    assert (x + 1).sum().item() == 16


def test_a_wait_for_words_that_runs_out_ends_its_own_launch_only():
    """The step without barriers: a wait that nothing serves raises the flag and returns; while the flag is up, a wait of another pair
    that takes some hundred looks is served all the same, and a model's step is what it was."""
    import ctypes
    assert healthy() == 0
    m, _, _ = small_lm("aspin", "rms", torch.bfloat16)
    ids = synth.token_ids(1, 40, 256, seed=5).to(DEV)

    def steps():
        dec = Decoder(m, batch=1)
        dec.prefill(ids[:, :36])
        out = torch.stack([dec.step(ids[:, t]).clone() for t in range(36, 40)])
        assert dec._plan["flow"]
        return out

    def wait(limit, late):
        words, sync = torch.zeros(128, dtype=torch.int32, device=DEV), torch.zeros(2, dtype=torch.int64, device=DEV)
        rc = _lib.lib().pgb_decode_flow_wait_selftest(ctypes.c_void_p(words.data_ptr()), ctypes.c_void_p(sync.data_ptr()), limit, late, None)
        assert rc == 0
        torch.cuda.synchronize()
        return words, sync.tolist()

    want = steps()
    words, sync = wait(2000, -1)
    assert sync == [1, 1] and not words.any()
    words, sync = wait(1 << 20, 1_000_000)                            # half a millisecond: far more than 64 looks
    assert sync == [1, 0] and bool((words >> 16 == 1).all())
    assert torch.equal(steps(), want)
    assert healthy() == 82 and healthy() == 0                         # reported once, then clear
    L, one = _lib.lib(), ctypes.c_void_p(16)
    assert L.pgb_decode_flow_wait_selftest(one, one, 0, 0, None) == 2 and L.pgb_decode_flow_wait_selftest(None, one, 1, 0, None) == 1
