"""The work a user of pragnosia_b200 has it do, as cases that can be timed and compared: language-model prefill with the
carried state, decoding after a prompt, and the operators under both (the associative scan with either write rule, the
per-token lambda scan), forward and -- where they are trained through -- backward.

    listed()            the fixed cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program has in hand before the call (weights, inputs, a Decoder)
    run(state)          one pass through the public entry points
    work(case)          the bytes and operations one pass cannot do without
    tolerance(case)     how far two correct implementations may lie apart

Sizes are those of the benchmark configurations and of the reference's own published measurements; everything is synthetic
(random-init weights, uniform token ids) with the distributions of pragnosia_b200/synth.py.
"""
import math

import torch
import torch.nn.functional as F

from pragnosia_b200 import synth
from pragnosia_b200.assoc import assoc_scan
from pragnosia_b200.assoc_kernel import assoc_scan_kernel, delta_scan_kernel, prep_kernel
from pragnosia_b200.generate import Decoder
from pragnosia_b200.model import LM
from pragnosia_b200.scan_kernel import scan_cuda

VOCAB, WIDTH, WINDOW = 8192, 768, 512                                 # the benchmark's language model (random init, bf16 weights)
DEV = "cuda"


def _layers(mixer):
    # Twelve, as the benchmark has it; six under the delta rule, whose random-init states drift apart by 3e-2 over twelve
    # layers between two implementations that only round one activation differently.
    return 6 if mixer in ("dspin", "hdspin") else 12


def listed():
    return [
        # A batch of prompts through the language model, four carried 512-token windows: the headline configuration.
        dict(name="lm_b16", kind="lm", mixer="aspin", B=16, T=2048),
        # One long prompt: a single user's context taken in, sixteen windows one behind the other.
        dict(name="lm_b1", kind="lm", mixer="aspin", B=1, T=8192),
        # A few prompts whose length is no whole number of windows (nor of 64-token chunks), with the delta write rule.
        dict(name="lm_ragged_delta", kind="lm", mixer="dspin", B=3, T=1333),
        # A single user's request: prompt, then tokens one at a time.
        dict(name="decode_b1", kind="decode", mixer="aspin", B=1, T=512, steps=64),
        # A server's batch of requests in step.
        dict(name="decode_b64", kind="decode", mixer="aspin", B=64, T=512, steps=64),
        # The operator in its precise fp32 mode, two short sequences: the smallest call.
        dict(name="scan_fp32", kind="scan", rule="plain", dtype="fp32", B=2, H=12, T=512, D=64),
        # One long-context window of 64 sequences, bf16, state carried in and out.
        dict(name="scan_plain", kind="scan", rule="plain", dtype="bf16", B=64, H=12, T=4096, D=64),
        # The delta rule at head dim 128 over a long sequence.
        dict(name="scan_delta", kind="scan", rule="delta", dtype="bf16", B=8, H=16, T=8192, D=128),
        # The diagonal carrier's scan over one long-context window, one rotation angle per token.
        dict(name="lambda_fwd", kind="lambda", angle="token", train=False, B=64, T=4096, D=768),
        # The same scan in training, forward and backward, one angle per channel (what the layer passes).
        dict(name="lambda_train", kind="lambda", angle="channel", train=True, B=16, T=512, D=704),
        # Training through the associative layer's operators (plumbing, then scan), forward and backward: both rules.
        dict(name="train_plain", kind="train", rule="plain", B=4, H=11, T=2048, D=64),
        dict(name="train_delta", kind="train", rule="delta", B=4, H=11, T=2048, D=64),
    ]


def _log(rng, lo, hi):
    """A whole number from lo..hi, spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["lm", "decode", "scan", "scan", "lambda", "train"])
    if kind == "lm":                                                  # whole windows and ragged lengths alike
        B = _log(rng, 1, 16)
        if rng.random() < 0.4:
            T = WINDOW * _log(rng, 1, min(16, 32768 // (B * WINDOW)))
        else:
            T = _log(rng, 64, min(8192, 32768 // B))
        return dict(kind=kind, mixer=rng.choice(["aspin", "aspin", "dspin", "hspin", "hdspin"]), B=B, T=T)
    if kind == "decode":
        return dict(kind=kind, mixer=rng.choice(["aspin", "aspin", "dspin"]), B=_log(rng, 1, 64), T=_log(rng, 16, 1024),
                    steps=rng.randint(16, 64))
    if kind == "scan":
        rule, D, dtype = rng.choice(["plain", "delta"]), rng.choice([64, 128]), rng.choice(["bf16", "bf16", "fp32"])
        B, H = _log(rng, 1, 64), rng.randint(2, 16)
        most = (1 << 17 if dtype == "fp32" else 1 << 20 if rule == "delta" else 3 << 20) * 64 // (B * H * D)
        return dict(kind=kind, rule=rule, dtype=dtype, B=B, H=H, T=_log(rng, 32, max(32, min(8192, most))), D=D)
    if kind == "lambda":
        train = rng.random() < 0.5
        B, D = _log(rng, 1, 64), _log(rng, 64, 1024)
        if rng.random() < 0.7:
            D = D // 4 * 4                                            # most widths are multiples of four; some are not
        most = ((16 * 512 * 768 * 4) if train else (64 * 4096 * 768)) // (B * D)
        return dict(kind=kind, angle=rng.choice(["token", "channel"]), train=train, B=B, T=_log(rng, 32, max(32, min(4096, most))), D=D)
    D = rng.choice([64, 128])
    B, H = _log(rng, 1, 8), rng.randint(2, 16)
    most = 4 * 11 * 2048 * 64 * 64 // (B * H * D * D)
    return dict(kind=kind, rule=rng.choice(["plain", "delta"]), B=B, H=H, T=_log(rng, 64, max(64, min(4096, most))), D=D)


def _language_model(mixer, seed):
    torch.manual_seed(seed)
    with torch.device(DEV):                                           # initialised where it will live
        m = LM(vocab=VOCAB, d=WIDTH, layers=_layers(mixer), mlp_mult=4, ctx=WINDOW, mixer=mixer, norm="rms")
    return m.to(torch.bfloat16).eval()


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=g)
    kind, B, T = case["kind"], case["B"], case["T"]
    if kind in ("lm", "decode"):
        m = _language_model(case["mixer"], seed)
        ids = torch.randint(0, VOCAB, (B, T), device=DEV, generator=g)
        if kind == "lm":
            return dict(case=case, model=m, ids=ids)
        # the continuation's tokens are given (scoring a text, constrained decoding), so that every implementation takes
        # the same ones
        return dict(case=case, decoder=Decoder(m, batch=B), ids=ids,
                    forced=torch.randint(0, VOCAB, (case["steps"], B), device=DEV, generator=g))
    if kind == "lambda":
        D = case["D"]
        logmag = (0.9 + 0.099 * torch.rand(B, T, D, device=DEV, generator=g)).log()
        if case["angle"] == "channel":
            ang = math.pi * torch.rand(D, device=DEV, generator=g)
        else:
            ang = math.pi * torch.rand(B, T, D, device=DEV, generator=g)
        st = dict(case=case, u=rn(B, T, D) * (0.1 * rn(D)), logmag=logmag, ang=ang, h0=(rn(B, D), rn(B, D)))
        if case["train"]:
            st["dy"] = rn(B, T, D)
            for n in ("u", "logmag", "ang"):
                st[n].requires_grad_(True)
        return st
    H, D = case["H"], case["D"]
    la = F.logsigmoid(2.0 + rn(B, H, T))
    beta = torch.sigmoid(rn(B, H, T)) if case["rule"] == "delta" else None
    if kind == "scan":
        dt = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
        q, k, v = rn(B, H, T, D).to(dt), F.normalize(rn(B, H, T, D), dim=-1).to(dt), rn(B, H, T, D).to(dt)
        return dict(case=case, q=q, k=k, v=v, la=la, beta=beta, S0=0.1 * rn(B, H, D, D))
    st = dict(case=case, la=la, beta=beta, theta=synth.rope_theta(H, D).to(DEV), pos=torch.arange(T, device=DEV),
              gate=None if beta is not None else rn(B, T, H).to(torch.bfloat16), do=rn(B, H, T, D).to(torch.bfloat16))
    for n in ("qp", "kp", "vp"):                                      # the projections' outputs, (B,T,H,D)
        st[n] = rn(B, T, H, D).to(torch.bfloat16)
    # The rotation frequencies stay fixed: their gradient weighs the absolute position while the result depends on relative
    # ones only, so q's and k's shares cancel down to the noise of bf16 operands (0.2-0.4 between two implementations).
    st["wrt"] = [n for n in ("qp", "kp", "vp", "gate", "la", "beta") if st[n] is not None]
    for n in st["wrt"]:
        st[n].requires_grad_(True)
    return st


def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind == "lm":
        logits, states = s["model"].forward_carried(s["ids"], WINDOW, return_states=True)
        return {"logits": logits, "states": [st[0] for st in states]}
    if kind == "decode":
        dec = s["decoder"]
        logits = torch.empty(case["steps"] + 1, case["B"], VOCAB, device=DEV)
        logits[0].copy_(dec.prefill(s["ids"]))
        for i, tok in enumerate(s["forced"].unbind(0)):
            logits[i + 1].copy_(dec.step(tok))
        return {"logits": logits, "states": [st[0] for st in dec.states]}
    if kind == "scan":
        with torch.no_grad():
            return assoc_scan(s["q"], s["k"], s["v"], s["la"], s["S0"], beta=s["beta"])
    if kind == "lambda":
        ang = s["ang"].expand_as(s["logmag"])
        if not case["train"]:
            with torch.no_grad():
                return scan_cuda(s["u"], s["logmag"], ang, s["h0"])
        with torch.enable_grad():
            y, (hr, hi) = scan_cuda(s["u"], s["logmag"], ang, s["h0"])
        return [y.detach(), hr.detach(), hi.detach(), *torch.autograd.grad(y, [s["u"], s["logmag"], s["ang"]], s["dy"])]
    with torch.enable_grad():
        q, k, v = prep_kernel(s["qp"], s["kp"], s["vp"], s["gate"], s["theta"], s["pos"])
        if s["beta"] is None:
            o, S, _ = assoc_scan_kernel(q, k, v, s["la"])
        else:
            o, S, _ = delta_scan_kernel(q, k, v, s["la"], s["beta"])
    return [o.detach(), S.detach(), *torch.autograd.grad(o, [s[n] for n in s["wrt"]], s["do"])]


def work(case):
    kind, B, T = case["kind"], case["B"], case["T"]
    if kind in ("lm", "decode"):
        D = 128 if case["mixer"] in ("hspin", "hdspin") else 64
        H = WIDTH // D
        per_layer = 12 * WIDTH * WIDTH + 2 * H * WIDTH                # q, k, v, o, the two gates, MLP up and down
        L = _layers(case["mixer"])
        weights, head = L * per_layer, VOCAB * WIDTH
        mix = L * (4 * 64 * WIDTH + 4 * D * WIDTH) * (2 if case["mixer"] in ("dspin", "hdspin") else 1)
        state = L * B * H * D * D * 4
        if kind == "lm":
            last = (T - 1) % WINDOW + 1
            return {"bytes": 2 * (weights + head) + 8 * B * T + 2 * B * last * VOCAB + state,
                    "flops": B * T * (2 * weights + mix) + 2 * B * last * head}
        n = case["steps"]
        # the weights do not fit in the caches with the states, so every step reads them
        return {"bytes": 2 * (weights + head) + 8 * B * T + n * (2 * (weights + head) + 2 * state + 4 * B * VOCAB),
                "flops": B * T * (2 * weights + mix) + 2 * B * head + n * B * (2 * (weights + head) + L * 4 * D * WIDTH)}
    if kind == "lambda":
        n, D = B * T * case["D"], case["D"]
        a = n if case["angle"] == "token" else D
        fwd = 4 * (3 * n + a + 4 * B * D)
        if not case["train"]:
            return {"bytes": fwd, "flops": 10 * n}
        # the backward reads the inputs, the states and dy again and writes a gradient for each input
        return {"bytes": fwd + 4 * (6 * n + 2 * a), "flops": 40 * n}
    H, D = case["H"], case["D"]
    rows, delta = B * H * T, case["rule"] == "delta"
    per_row = (8 * 64 * D + 6 * D * D + 64 * 64) if delta else (4 * 64 * D + 4 * D * D)
    if kind == "scan":
        e = 2 if case["dtype"] == "bf16" else 4
        return {"bytes": rows * (4 * D * e + 4 * (1 + delta)) + 8 * B * H * D * D, "flops": rows * per_row}
    # q, k, v in, o out; then q, k, v and do in, dq, dk, dv out
    return {"bytes": rows * (11 * D * 2 + 12 * (1 + delta)) + 4 * B * H * D * D, "flops": 3 * rows * per_row}


def tolerance(case):
    kind = case["kind"]
    if kind in ("lm", "decode"):
        # bf16 residual stream and activations over the layers: another rounding of one activation moves the logits by
        # 1.7e-2 and the deepest states by 1e-2 to 2e-2
        return {"rel": 3e-2}
    if kind == "lambda":
        return {"rel": 1e-5}
    if kind == "scan":
        return {"rel": 1e-5} if case["dtype"] == "fp32" else {"rel": 5e-3}
    return {"rel": 1e-2}                                              # bf16 operands and gradients; the states between the operators are bf16
