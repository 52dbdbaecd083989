"""A few long chains of the plain rule cut into segments that run side by side, against the same call walking them whole (which an
in-place state takes) and against the chunked oracle."""
import pytest
import torch

import oracle.carrier_oracle as oracle
from pragnosia_b200 import _lib, ops, synth

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


@pytest.mark.parametrize("B,H,T", [(1, 1, 1024), (1, 2, 1025), (2, 6, 2048), (4, 11, 2047), (1, 12, 8192), (1, 1, 20000), (1, 74, 2817),
                                   (13, 12, 1100), (150, 2, 1090), (25, 12, 2050)])   # the last round's only
@pytest.mark.parametrize("shift", [0.0, 37.0])
def test_segments_match_the_whole_walk(B, H, T, shift):
    assert _lib.lib().pgb_aspin_prefill_segments_scratch_bytes(B, H, T, 64) > 0
    g = torch.Generator(device="cuda").manual_seed(T)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k, v = rn(B, H, T, 64).bfloat16(), torch.nn.functional.normalize(rn(B, H, T, 64), dim=-1).bfloat16(), rn(B, H, T, 64).bfloat16()
    la, S0, th = -0.02 * torch.rand(B, H, T, device="cuda", generator=g), rn(B, H, 64, 64), synth.rope_theta(H, 64).cuda()
    o, S, sent = ops.prefill(q, k, v, la, S0=S0, theta=th, shift=shift, want_sent=True)
    inplace = S0.clone()
    o1, S1, sent1 = ops.prefill(q, k, v, la, S0=inplace, theta=th, shift=shift, want_sent=True, S_out=inplace)
    assert rel(o, o1) < 1e-3 and rel(S, S1) < 1e-5 and rel(sent, sent1) < 1e-3
    if shift == 0.0 and T <= 2048:
        for s0 in (None, S0):
            ro, rS = oracle.assoc_scan(*(t.float().cpu() for t in (q, k, v, la)), None if s0 is None else s0.cpu())
            o, S, _ = ops.prefill(q, k, v, la, S0=s0)
            assert rel(o.cpu(), ro) < 4e-3 and rel(S.cpu(), rS) < 1e-4


@pytest.mark.parametrize("B,H,T,D", [(1, 1, 960, 64), (1, 75, 4096, 64), (1, 2, 4096, 128), (3, 100, 4096, 64), (13, 12, 960, 64), (20, 10, 4096, 64)])
def test_not_worth_cutting(B, H, T, D):
    assert _lib.lib().pgb_aspin_prefill_segments_scratch_bytes(B, H, T, D) == 0
