"""The fp32 plain prefill in groups of bounded scratch, and without any, against the chain-by-chain walk of the same arithmetic."""
import pytest
import torch

from pragnosia_b200 import _lib, ops, synth

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def operands(B, H, T, D, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=g)
    k = rn(B, H, T, D)
    k /= k.norm(dim=-1, keepdim=True)
    return rn(B, H, T, D), k, rn(B, H, T, D), -0.05 * torch.rand(B, H, T, device=DEV, generator=g), rn(B, H, D, D), synth.rope_theta(H, D).to(DEV)


def walk(q, k, v, la, S0, theta, shift):
    B, H, T, D = q.shape
    o, S = torch.empty_like(q), torch.empty_like(S0)
    sent = torch.empty(B, H, (T + 63) // 64, D, D, device=DEV, dtype=torch.bfloat16)
    p = _lib.ptr
    _lib.check(_lib.lib().pgb_aspin_prefill_fwd(p(q), p(k), p(v), _lib.F32, p(la), None, p(S0), p(theta), None, shift, p(o), _lib.F32, p(S), p(sent), B, H, T, D,
                                                _lib.PREFILL_AUTO, torch.cuda.current_stream().cuda_stream), "pgb_aspin_prefill_fwd")
    return o, S, sent


# groups of two batch rows and a last one, of some heads of a row, of pieces of one chain; one chunk a chain, few and many of them
@pytest.mark.parametrize("B,H,T,D", [(5, 4, 1100 * 64 - 7, 64), (2, 5, 1700 * 64 + 1, 64), (1, 2, 4097 * 64 + 5, 128), (1, 1, 16385 * 64, 64), (2, 3, 64, 64),
                                     (10, 12, 50, 64), (10, 12, 64, 128)])
def test_groups_match_the_walk(B, H, T, D):
    x = operands(B, H, T, D, T)
    peak = torch.cuda.max_memory_allocated
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    got = ops.prefill(*x[:4], S0=x[4], theta=x[5], shift=33.0, want_sent=True)
    kept = sum(t.numel() * t.element_size() for t in got)
    assert peak() - before - kept <= (256 << 20) + (1 << 20)
    for a, b, tol in zip(got, walk(*x, 33.0), (1e-5, 1e-5, 1e-3)):    # sums in another order; the chunks' states rounded to bf16
        assert rel(a, b) < tol
    S = x[4].clone()
    o, S1, _ = ops.prefill(*x[:4], S0=S, theta=x[5], shift=33.0, S_out=S)        # in place
    assert S1 is S or S1.data_ptr() == S.data_ptr()
    assert torch.equal(S, got[1]) and torch.equal(o, got[0])


def test_walks_where_the_scratch_cannot_be_had():
    x = operands(1, 16, 16384, 128, 1)                                # o 134 MB, scratch 268
    want = ops.prefill(*x[:4], S0=x[4])[:2]
    torch.cuda.synchronize(); torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (200 << 20)) / total)
    try:
        got = ops.prefill(*x[:4], S0=x[4])[:2]
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert all(rel(a, b) < 1e-5 for a, b in zip(got, want))
