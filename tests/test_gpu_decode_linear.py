"""The decode step of a batch as a chain of dependent launches (decode_linear.cu) against the same step through the separate kernels, whose
parity with the oracle the model tests pin. Both round after every linear layer, norm, activation and add; the chain applies a norm's
1 / rms to the fp32 sum instead of the row ahead of it and adds a product's K in parts, so a bf16 rounding may fall the other way
(2^-8 of a value). So both are measured against the same model in fp32 (weights of the same values): the 2-norm of the chain's error is that
of the separate kernels', as two draws of the same roundings (measured 0.95 to 1.07 of it)."""
import copy

import pytest
import torch
import torch.nn.utils.parametrize

from pragnosia_b200 import _lib, ops, synth
from pragnosia_b200.assoc import AssocCarrier
from pragnosia_b200.generate import Decoder
from pragnosia_b200.model import LM

from test_gpu_decode_token import healthy
from test_gpu_model import DEV

pytestmark = pytest.mark.gpu


def model(d, mixer, mult, vocab, layers=3, norm="rms"):
    torch.manual_seed(d)
    m = LM(vocab=vocab, d=d, layers=layers, mlp_mult=mult, ctx=16, mixer=mixer, norm=norm)
    with torch.no_grad():
        for n, p in m.named_parameters():
            if p.dim() == 1:                                          # norms' weights, biases, gates: away from their initial ones and zeros
                p.add_(0.2 * torch.randn_like(p))
    return m.to(DEV).bfloat16().eval()


def steps(m, B, vocab, n=10, **kw):
    ids = synth.token_ids(B, 40, vocab, seed=B).to(DEV)
    dec = Decoder(m, batch=B, **kw)
    lg = [dec.prefill(ids[:, :20])]
    for t in range(20, 20 + n):                                       # crosses the window's edge (ctx 16)
        lg.append(dec.step(ids[:, t]).clone())
    lg.append(dec.prefill(ids[:, :17]))                               # a new prompt on the same decoder
    lg.append(dec.step(ids[:, 17]).clone())
    return dec, torch.stack(lg, 1), [st[0].clone() for st in dec.states]


@pytest.mark.parametrize("d,mixer,mult,vocab", [
    (256, "hspin", 1, 40),                                            # the least K, clusters of two; a head of one tile; head dim 128
    (704, "dspin", 3, 1000),                                          # eleven blocks over two and four CTAs, 33 over eight; ragged tiles of every width
    (768, "aspin", 4, 8192),
    (1536, "hdspin", 4, 5000),                                        # twelve blocks a CTA
])
@pytest.mark.parametrize("B", [5, 16, 17, 44, 64])
def test_chained_step_of_a_batch(d, mixer, mult, vocab, B):
    m = model(d, mixer, mult, vocab)
    _, lg_x, S_x = steps(copy.deepcopy(m).float(), B, vocab)
    ref, lg0, S0 = steps(m, B, vocab, fused=False)
    assert not ref._chain_ok()
    off = lambda lg, S: [float((a.double() - x.double()).norm() / x.double().norm()) for a, x in zip((lg, *S), (lg_x, *S_x))]
    outs = []
    for use_graph in (True, False):
        dec, lg, S = steps(m, B, vocab, use_graph=use_graph)
        assert dec._chain_ok() and dec.launches_per_token == 3 + 5 * m.layers
        assert all(torch.isfinite(t).all() for t in (lg, *S))
        ratios = [e / e0 for e, e0 in zip(off(lg, S), off(lg0, S0))]
        assert max(ratios) < 1.2
        outs.append((lg, S))
    assert torch.equal(outs[0][0], outs[1][0]) and all(torch.equal(a, b) for a, b in zip(outs[0][1], outs[1][1]))   # every sum in a fixed order
    assert healthy() == 0


def test_models_that_keep_the_separate_kernels():
    for m, B, kw in ((model(192, "aspin", 2, 256), 8, {}), (model(256, "aspin", 2, 256, norm="ln"), 8, {}), (model(256, "aspin", 2, 256), 65, {}), (model(256, "aspin", 2, 256), 8, dict(folded=True)),
                     (model(256, "aspin", 2, 252), 8, {})):
        dec, lg, _ = steps(m, B, 250, n=2, **kw)
        assert not dec._chain_ok() and torch.isfinite(lg).all()


def test_generate_through_the_chained_step():
    m = model(256, "aspin", 4, 512)
    prompt = synth.token_ids(9, 40, 512, seed=3).to(DEV)
    for temp in (0.0, 1.0):
        a = Decoder(m, batch=9).generate(prompt, 24, temp=temp, seed=5)
        c = Decoder(m, batch=9, use_graph=False).generate(prompt, 24, temp=temp, seed=5)
        assert torch.equal(a, c)                                      # graph replay and eager launches draw the same ids
    assert healthy() == 0


@pytest.mark.parametrize("K", [6656, 6720, 7168, 7680])               # the longest rows of the wider tiles, the shortest and longest past them
@pytest.mark.parametrize("B", [5, 32, 33, 64])
def test_long_rows_of_a_residual_layer(K, B):
    """Against 64 bits: v is rounded to bf16 and so is resid + v (2^-9 of each); the products' sums are fp32 (K 2^-24 of the sum of magnitudes at most)."""
    g = torch.Generator(device=DEV).manual_seed(K + B)
    N = 136                                                           # ragged tiles of 32 and of 48 columns
    x, W, r, w = (torch.randn(*s, device=DEV, generator=g).bfloat16() for s in ((B, K), (N, K), (B, N), (N,)))
    y, yw, sq = ops.decode_linear(x, W, resid=r, next_w=w)
    v = x.double() @ W.double().T
    slack = 2.0 ** -24 * K * (x.double().abs() @ W.double().abs().T)
    want = v + r.double()
    assert bool(((y.double() - want).abs() <= 2.0 ** -9 * 1.01 * (v.abs() + want.abs() + 2.0 ** -8 * v.abs()) + 2 * slack).all())
    assert torch.equal(yw, (y.float() * w.float()).bfloat16())
    torch.testing.assert_close(sq.double().sum(1), y.double().square().sum(1), rtol=2.0 ** -24 * 64, atol=0)     # sums of 136 squares in fp32
    assert healthy() == 0


class HalfCarrier(AssocCarrier):
    def mix(self, z, h0=None, inplace=None):
        delta, st = super().mix(z, h0, inplace)
        return 0.5 * delta, st


class OwnNorm(torch.nn.RMSNorm):
    pass


def test_layers_of_other_types_keep_their_own_step():
    """The chain calls kernels, not the layers: a carrier with a mix of its own, and norms and tables whose type may form their weight as it is
    asked for (the chain's kernels read weights ahead of their waits), stay with the separate kernels."""
    ids = synth.token_ids(8, 30, 256, seed=1).to(DEV)
    for change in ("mix", "norm", "table"):
        m = model(256, "aspin", 2, 256)
        if change == "mix":
            m.mix[1].__class__ = HalfCarrier
        elif change == "norm":
            m.mlp[0].n.__class__ = OwnNorm
        else:
            torch.nn.utils.parametrize.register_parametrization(m.e, "weight", torch.nn.Identity())
        outs = []
        for fused in (True, False):
            dec = Decoder(m, batch=8, fused=fused, use_graph=False)
            dec.prefill(ids[:, :20])
            outs.append([dec.step(ids[:, t]).clone() for t in range(20, 24)])
            assert not dec._chain_ok()
        assert all(torch.equal(a, b) for a, b in zip(*outs)), change


@pytest.mark.parametrize("d,mixer,B", [(704, "dspin", 17), (768, "aspin", 44)])          # an odd number of pairs: the last CTA has one
def test_chained_step_with_a_warp_per_pair(d, mixer, B):
    """The chain takes a CTA per pair of its own accord; where the other kernel is asked for, it reads its state ahead of the wait, too."""
    L = _lib.lib()
    _lib.check(L.pgb_decode_set_variant(2), "pgb_decode_set_variant")
    try:
        test_chained_step_of_a_batch(d, mixer, 3, 1000, B)
    finally:
        _lib.check(L.pgb_decode_set_variant(0), "pgb_decode_set_variant")


def between(y, want, slack, then=lambda t: t):
    """Rounding is monotone: y = then(bf16(fp32 sum)) lies between what the ends of the sum's interval give."""
    return bool(((y >= then((want - slack).bfloat16())) & (y <= then((want + slack).bfloat16()))).all())


@pytest.mark.parametrize("N,K,tile", [(1080, 3256, 48), (568, 4600, 48), (2104, 2104, 64), (760, 6136, 64), (2168, 2168, 96), (1080, 4344, 96)])
def test_tiles_of_wide_residual_layers(N, K, tile):
    """Links that take more than one round in the first form: tiles and clusters of the others, N and K ragged. The fp32 sum is within K 2^-24 of the sum of
    magnitudes; v, then resid + v, are rounded to bf16."""
    B = 64
    assert _lib.lib().pgb_decode_linear_parts(N, K, B) == -(-N // tile)
    g = torch.Generator(device=DEV).manual_seed(N)
    x, W, r, w = (torch.randn(*s, device=DEV, generator=g).bfloat16() for s in ((B, K), (N, K), (B, N), (N,)))
    y, yw, sq = ops.decode_linear(x, W, resid=r, next_w=w)
    v = x.double() @ W.double().T
    assert between(y, v, 2.0 ** -24 * K * (x.double().abs() @ W.double().abs().T), lambda t: (t.float() + r.float()).bfloat16())
    assert torch.equal(yw, (y.float() * w.float()).bfloat16())
    torch.testing.assert_close(sq.double().sum(1), y.double().square().sum(1), rtol=2.0 ** -24 * 64, atol=0)
    assert healthy() == 0


@pytest.mark.parametrize("N,K", [(1976, 1976), (3832, 952), (2104, 2104), (4664, 4664), (6008, 1976), (3896, 3896)])     # 32 x 4, 64 x 2, 4 and 8, 96 x 4 and 8
@pytest.mark.parametrize("B", [5, 64])
def test_tiles_of_wide_layers_behind_a_norm(N, K, B):
    """v = r (x W^T) + bias, rounded to bf16 once; r is off by its sum, division and root, each in fp32 (2^-20 covers them)."""
    g = torch.Generator(device=DEV).manual_seed(N + B)
    x, W, b = (torch.randn(*s, device=DEV, generator=g).bfloat16() for s in ((B, K), (N, K), (N,)))
    sq = torch.rand(B, 24, device=DEV, generator=g) * K
    y = ops.decode_linear(x, W, b, sq, 1e-5)
    rs = (sq.double().sum(1, keepdim=True) / K + 1e-5).rsqrt()
    v = rs * (x.double() @ W.double().T)
    slack = rs * 2.0 ** -24 * K * (x.double().abs() @ W.double().abs().T) + 2.0 ** -20 * v.abs() + 2.0 ** -24 * b.double().abs()
    assert between(y, v + b.double(), slack)
    assert healthy() == 0


@pytest.mark.parametrize("d,mult,B,taken", [(1664, 4, 48, True), (1664, 4, 49, False), (1536, 4, 64, True), (2304, 3, 8, True), (2304, 3, 9, False), (3072, 2, 5, False)])
def test_wide_models_whose_links_take_many_rounds(d, mult, B, taken):
    """The chain where it is the quicker, the separate kernels elsewhere: by the rounds of a layer's links and the batch."""
    m = model(d, "aspin", mult, 256, layers=1)
    assert Decoder(m, batch=B)._chain_ok() == taken
