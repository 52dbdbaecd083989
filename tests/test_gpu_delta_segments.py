"""The delta rule with few chains, segments side by side (delta_segments.cu), against the same call given the inverses' scratch only, which walks every
chain as a whole. Each is 5.2e-6 (o) and 3.6e-6 (S) from 64 bits in the 2-norm, so the two lie within the sums of those."""
import ctypes

import pytest
import torch
import torch.nn.functional as F

from pragnosia_b200 import _lib, ops

pytestmark = pytest.mark.gpu
torch.set_grad_enabled(False)
DEV = "cuda"


@pytest.mark.parametrize("B,H,T", [(3, 12, 1333), (1, 2, 2048), (1, 12, 4000), (1, 5, 1025), (2, 3, 700), (1, 40, 2048), (1, 1, 8192)])
@pytest.mark.parametrize("S0,shift", [(False, 0.0), (True, 0.0), (True, 37.0)])
def test_segments_side_by_side_match_whole_chains(B, H, T, S0, shift):
    D, L = 64, _lib.lib()
    g = torch.Generator(device=DEV).manual_seed(T + H)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=g)
    q, k, v = rn(B, H, T, D).bfloat16(), F.normalize(rn(B, H, T, D), dim=-1).bfloat16(), rn(B, H, T, D).bfloat16()
    la, beta, th = F.logsigmoid(2.0 + rn(B, H, T)), torch.sigmoid(rn(B, H, T)), rn(H, D // 2).abs()
    S_in = rn(B, H, D, D) if S0 else None
    n = L.pgb_aspin_delta_scratch_bytes(B, H, T)
    assert L.pgb_aspin_delta_prefill_scratch_bytes(B, H, T, D) > n                       # these are cut
    p = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None
    whole = [torch.empty(B, H, T, D, device=DEV), torch.empty(B, H, D, D, device=DEV)]
    x = torch.empty(n, device=DEV, dtype=torch.uint8)
    assert L.pgb_aspin_delta_prefill_fwd(p(q), p(k), p(v), p(la), p(beta), p(S_in), p(th), None, shift, p(whole[0]), 0, p(whole[1]), None, p(x), n, B, H, T, D,
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    o, S, _ = ops.prefill(q, k, v, la, beta, S_in, theta=th, shift=shift, out_dtype=torch.float32)
    rel = lambda a, b: float((a.double() - b.double()).norm() / b.double().norm())
    assert rel(o, whole[0]) <= 1.1e-5 and rel(S, whole[1]) <= 7.5e-6, (rel(o, whole[0]), rel(S, whole[1]))
    ob, Sb, _ = ops.prefill(q, k, v, la, beta, S_in, theta=th, shift=shift)
    assert torch.equal(ob, o.bfloat16()) and torch.equal(Sb, S)                          # the bf16 read is the fp32 one, rounded


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("half", [16, 32])                            # the join of 16-wide blocks, and that of 32-wide ones
def test_joins_of_the_chunk_inverse_keep_fp32(D, half):
    """Tokens s < t < u of one unit key, no decay: N[t][s] = b_t, N[u][s] = N[u][t] = b_u, all 24 bits of them, and X[u][s] = -b_u + b_u b_t, which for b_t just
    below 1 cancels down to the factors' last bits. In fp32 the one rounding of b_u b_t is 2^-25 of b_u, and the pair of bf16 it is stored as misses 2^-17 of a
    result below 2^-8: 2^-24 in all. Factors as two tf32 parts: up to 2^-22.5 (emulated; they were taken back)."""
    n, L = half // 2, _lib.lib()                                      # triples a chunk: s = i in the upper block, t and u neighbours in the lower
    B, H, NC = 1, 4, 64
    T = 64 * NC
    own = torch.arange(64)
    for i in range(n):
        own[half + 2 * i] = own[half + 2 * i + 1] = i
    k = F.one_hot(own, D).bfloat16().to(DEV).repeat(B * H * NC, 1, 1).view(B, H, T, D)
    g = torch.Generator(device=DEV).manual_seed(half)
    beta = 0.5 + 0.5 * torch.rand(B, H, NC, 64, device=DEV, generator=g)
    s, t = torch.arange(n, device=DEV), half + 2 * torch.arange(n, device=DEV)
    beta[..., t] = 1 - (1 + torch.rand(B, H, NC, n, device=DEV, generator=g)) * 2.0 ** -9
    q, v, la = torch.zeros_like(k), torch.zeros_like(k), torch.zeros(B, H, T, device=DEV)
    p = lambda a: ctypes.c_void_p(a.data_ptr())
    x = torch.empty(L.pgb_aspin_delta_scratch_bytes(B, H, T), device=DEV, dtype=torch.uint8)
    o, S = torch.empty(B, H, T, D, device=DEV), torch.empty(B, H, D, D, device=DEV)
    assert L.pgb_aspin_delta_prefill_fwd(p(q), p(k), p(v), p(la), p(beta), None, None, None, 0.0, p(o), 0, p(S), None, p(x), x.numel(), B, H, T, D,
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    X = x[:B * H * NC * 2 * 8192].view(torch.bfloat16).view(B, H, NC, 2, 64, 64).double().sum(3)        # head + tail
    bt, bu = beta[..., t].double(), beta[..., t + 1].double()
    off = (X[..., t + 1, s] - (bu * bt - bu)).abs() / bu
    assert float(off.max()) <= 2.0 ** -24, float(off.max().log2())


@pytest.mark.parametrize("entry", ["prefill", "layer"])
def test_segments_whose_memory_cannot_be_had(entry):
    """Room for the inverses but not for the segments' share: the chains are walked whole, as a call with the least scratch walks them."""
    B, H, T, D, L = 1, 12, 16000, 64, _lib.lib()
    g = torch.Generator(device=DEV).manual_seed(3)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=g)
    if entry == "prefill":
        q, k, v = rn(B, H, T, D).bfloat16(), F.normalize(rn(B, H, T, D), dim=-1).bfloat16(), rn(B, H, T, D).bfloat16()
        la, beta = F.logsigmoid(2.0 + rn(B, H, T)), torch.sigmoid(rn(B, H, T))
        full, least = L.pgb_aspin_delta_prefill_scratch_bytes(B, H, T, D), L.pgb_aspin_delta_scratch_bytes(B, H, T)
        call = lambda: ops.prefill(q, k, v, la, beta)[:2]
    else:
        y, A, onw = rn(B, T, 3 * H * D + 2 * H).bfloat16(), torch.linspace(-2, -8, H, device=DEV), torch.ones(D, device=DEV)
        qp, kp, vp = (y[..., i * H * D:(i + 1) * H * D].unflatten(-1, (H, D)) for i in range(3))
        a, b, th, pos = y[..., 3 * H * D:3 * H * D + H], y[..., 3 * H * D + H:], rn(H, D // 2).abs(), torch.arange(T, device=DEV) % 512
        full, least = L.pgb_aspin_delta_layer_scratch_bytes(B, H, T, D), L.pgb_aspin_delta_layer_scratch_least_bytes(B, H, T, D)
        call = lambda: ops.delta_layer_windows(qp, kp, vp, a, b, A, th, pos, 512, onw, 1e-6)
    assert full > least + (64 << 20)
    want = call()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    ooms = torch.cuda.memory_stats()["num_ooms"]
    room = least + B * H * T * D * 2 + (32 << 20)
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + room) / torch.cuda.get_device_properties(0).total_memory)
    try:
        got = call()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.cuda.memory_stats()["num_ooms"] == ooms + 1
    rel = lambda x, y: float((x.double() - y.double()).norm() / y.double().norm())
    assert rel(got[0], want[0]) <= 2.0 ** -8 and rel(got[1], want[1]) <= 7.5e-6         # o is rounded to bf16 either way
