"""The lambda scan at the edges of what it takes: log-magnitudes whose exponential is zero, subnormal, infinite or NaN."""
import math

import pytest
import torch

from pragnosia_b200.scan_kernel import scan_cuda

pytestmark = pytest.mark.gpu


def literal(u, lm, an, h0=None):
    """The recurrence in fp64, token by token."""
    u, lm, an = u.double(), lm.double(), an.double().expand_as(lm)
    lam = torch.polar(lm.exp(), an)
    h = torch.zeros_like(u[:, 0], dtype=torch.complex128) if h0 is None else torch.complex(h0[0].double(), h0[1].double())
    out = []
    for t in range(u.shape[1]):
        h = lam[:, t] * h + u[:, t]
        out.append(h)
    return torch.stack(out, 1)


def rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


@pytest.mark.parametrize("train", [False, True])
@pytest.mark.parametrize("D", [8, 6, 3])
@pytest.mark.parametrize("T", [1, 37, 400])
@pytest.mark.parametrize("channel", [False, True])
def test_log_magnitudes_out_of_range(D, T, channel, train):
    """-inf is a reset (lambda = 0 exactly, whatever the state), results below the normal range are as small as they are, +inf and
    overflow are infinite, NaN stays NaN; each only where it reaches."""
    B = 2
    g = torch.Generator(device="cuda").manual_seed(D + T)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    u, lm, h0 = rn(B, T, D), -0.1 * rn(B, T, D).abs(), (1e30 * rn(B, D), 1e30 * rn(B, D))
    an = math.pi * torch.rand(D, device="cuda", generator=g)
    an = an.expand(B, T, D) if channel else an + 0.1 * rn(B, T, D)
    lm[:, 0] = float("-inf")                                          # forgets a state of 1e30: with the least magnitude that is not zero, 1e-8 of it stayed
    if T > 5:
        lm[:, 5] = -100.0                                             # e^-100 is subnormal
    if T > 30:
        lm[0, 30, 0] = float("inf")
        lm[1, 30, 0] = 200.0
        lm[0, 30, 1] = float("nan")
    with torch.enable_grad() if train else torch.no_grad():
        y, (hr, hi) = scan_cuda(u.requires_grad_(train), lm, an, h0)
    y, hr, hi = y.detach(), hr.detach(), hi.detach()
    h = literal(u.detach(), lm.float(), an, (torch.zeros(B, D, device="cuda"), torch.zeros(B, D, device="cuda")))
    bad = torch.zeros(B, T, D, dtype=torch.bool, device="cuda")
    if T > 30:
        bad[:, 30:, 0] = True
        bad[0, 30:, 1] = True
        assert not torch.isfinite(y[0, 30:, 0]).any() and not torch.isfinite(y[1, 30:, 0]).any() and torch.isnan(y[0, 30:, 1]).all()
    assert torch.isfinite(y[~bad]).all()
    assert rel(y[~bad], h.real[~bad]) < 1e-5
    last = ~bad[:, -1]
    assert rel(hr[last], h.real[:, -1][last]) < 1e-5 and (T < 2 or rel(hi[last], h.imag[:, -1][last]) < 1e-5)
    if T == 1:
        assert torch.equal(hr, u[:, 0].detach()) and not hi.any()
