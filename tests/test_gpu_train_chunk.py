"""The fused backward of the chunked scan (train_chunk.cu) through the drop-in names, against autograd through the CPU oracle
in fp64: one token, one whole chunk, a ragged last chunk, several chunks; both rules and head dims; a gradient on each of
the three results (outputs, final state, the states entering the chunks)."""
import pytest
import torch

import oracle
from pragnosia_b200 import assoc_kernel, synth

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize("delta", [False, True])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("T", [1, 64, 130, 333])
def test_fused_backward_matches_autograd_through_the_oracle(delta, D, T):
    B, H = 2, 3
    x = synth.assoc_op_inputs(B, H, T, D, seed=T + D, delta=True, with_state=True)
    g = torch.Generator().manual_seed(1)
    w_o = torch.randn(B, H, T, D, generator=g).to(torch.bfloat16)
    w_s, w_e = torch.randn(B, H, D, D, generator=g) * 0.1, torch.randn(B, H, (T + 63) // 64, D, D, generator=g) * 0.1
    names = ["q", "k", "v", "la", "S0"] + (["beta"] if delta else [])
    with torch.enable_grad():
        ref = {n: (x[n].to(torch.bfloat16) if n in "qkv" else x[n]).double().requires_grad_(True) for n in names}
        be = ref.get("beta")
        o_r, S_r = oracle.assoc_scan(ref["q"], ref["k"], ref["v"], ref["la"], ref["S0"], beta=be)
        loss = (o_r * w_o.double()).sum() + (S_r * w_s).sum()
        for c in range((T + 63) // 64):                               # the state entering chunk c: the scan of what is before it
            n = 64 * c
            S_c = ref["S0"] if c == 0 else oracle.assoc_scan(*(ref[m][:, :, :n] for m in ("q", "k", "v", "la")), ref["S0"],
                                                             beta=None if be is None else be[:, :, :n])[1]
            loss = loss + (S_c * w_e[:, :, c]).sum()
        loss.backward()
        dev = {n: (x[n].to(torch.bfloat16) if n in "qkv" else x[n]).cuda().requires_grad_(True) for n in names}
        args = [dev[n] for n in ("q", "k", "v", "la")] + ([dev["beta"]] if delta else []) + [dev["S0"]]
        o, S, sent = (assoc_kernel.delta_scan_kernel if delta else assoc_kernel.assoc_scan_kernel)(*args)
        ((o.float() * w_o.cuda().float()).sum() + (S * w_s.cuda()).sum() + (sent.float() * w_e.cuda()).sum()).backward()
    assert rel(o.detach().cpu(), o_r.detach()) <= 3e-3 and rel(S.detach().cpu(), S_r.detach()) <= 1e-5
    for n in names:                                                   # bf16 gradients; the saved states are bf16 as the operators keep them
        assert rel(dev[n].grad.cpu(), ref[n].grad) <= 4e-3, (n, rel(dev[n].grad.cpu(), ref[n].grad))


def _training_calls():
    g = torch.Generator(device="cuda").manual_seed(5)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k, v = (torch.nn.functional.normalize(rn(2, 3, 100, 64), dim=-1).bfloat16().requires_grad_() for _ in range(3))
    la, be = (-0.1 * torch.rand(2, 3, 100, device="cuda")).requires_grad_(), torch.rand(2, 3, 100, device="cuda").requires_grad_()
    qp, kp, vp = (rn(2, 100, 3, 64).bfloat16().requires_grad_() for _ in range(3))
    th, pos = torch.rand(3, 32, device="cuda"), torch.arange(100, device="cuda")
    return {"plain": (assoc_kernel.assoc_scan_kernel, (q, k, v, la), ("prefix_scan", "assoc_out")),
            "delta": (assoc_kernel.delta_scan_kernel, (q, k, v, la, be), ("delta_inv", "delta_loop_fwd", "assoc_out")),
            "prep": (lambda *x: (sum(assoc_kernel.prep_kernel(*x, None, th, pos)),), (qp, kp, vp), ("assoc_prep",))}


@pytest.mark.parametrize("what", ["plain", "delta", "prep"])
@torch.enable_grad()
def test_a_tracer_sees_operators(what):
    """make_fx of an eager training call records the registered operators; run without them the graph would hold the traced call's
    results as constants."""
    from torch.fx.experimental.proxy_tensor import make_fx
    f, args, ops_seen = _training_calls()[what]
    w = torch.randn(2, 3, 100, 64, device="cuda")
    gm = make_fx(lambda *x: torch.autograd.grad((f(*x)[0].float() * w).sum(), x))(*args)
    code = gm.code
    assert all(f"pragnosia_b200.{n}" in code for n in ops_seen)
    other = [(a.detach() * 0.5).requires_grad_() for a in args]
    want = torch.autograd.grad((f(*other)[0].float() * w).sum(), other)
    for a, b in zip(gm(*other), want):                                # the composition against the fused form: bf16 states between the operators
        assert rel(a.detach(), b) < 1e-2


@pytest.mark.parametrize("what", ["plain", "delta", "prep"])
@torch.enable_grad()
def test_a_second_differentiation_raises(what):
    """A gradient penalty over these operators is an error, not a loss without its gradient; a first derivative under create_graph is
    what it is without."""
    f, args, _ = _training_calls()[what]
    w = torch.randn(2, 3, 100, 64, device="cuda")
    want = torch.autograd.grad((f(*args)[0].float() * w).sum(), args)
    got = torch.autograd.grad((f(*args)[0].float() * w).sum(), args, create_graph=True)
    assert all(torch.equal(a.detach(), b) for a, b in zip(got, want))
    for g in got:
        with pytest.raises(RuntimeError, match="Trying to backward through"):
            torch.autograd.grad(g.float().square().sum() + f(*args)[0].float().sum(), args, retain_graph=True)


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("B,H,T,D", [(1, 1, 1, 64), (2, 3, 130, 64), (1, 2, 2048, 64), (1, 4, 1025, 64), (2, 3, 200, 128), (1, 2, 1024, 128)])
def test_the_final_state_of_training_is_fp32s(B, H, T, D, variant):
    """The plain rule's state against fp64 on the same bf16 operands: fp32 sums (64-token products, then the chunks) stay below 8e-7,
    scaled keys in two bf16 terms alone are 2e-6 off."""
    from pragnosia_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(T)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k, v = (torch.nn.functional.normalize(rn(B, H, T, D), dim=-1).bfloat16() for _ in range(3))
    la, S0 = torch.nn.functional.logsigmoid(2.0 + rn(B, H, T)), 0.1 * rn(B, H, D, D)
    L = la.double().cumsum(-1)
    want = (k.double() * (L[..., -1:] - L).exp()[..., None]).transpose(-1, -2) @ v.double() + L[..., -1].exp()[..., None, None] * S0.double()
    try:
        assert _lib.lib().pgb_tc_set_variant(variant) == 0
        S = ops.scan_train_fwd(q, k, v, la, None, S0)[1]
    finally:
        _lib.lib().pgb_tc_set_variant(0)
    assert rel(S, want) < 8e-7
