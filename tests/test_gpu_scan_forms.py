"""The forms the lambda scan, the prep backward and the fp32 chunked prefill choose between, at the edges of their ranges, against
the fp64 definitions: lanes of 4, 2 or 1 channels, tiles through slots in shared memory and through registers, angles past the range
of the fast sin/cos; rows read 16 bytes at a time or not."""
import pytest
import torch

import oracle.carrier_oracle as oracle
from pragnosia_b200 import _lib, ops, synth
from pragnosia_b200._lib import PREFILL_FP32

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


@pytest.mark.parametrize("B,T,D", [(1, 1, 4), (2, 7, 6), (3, 65, 5), (1, 129, 8), (700, 9, 512), (5, 257, 64), (2, 33, 301)])
@pytest.mark.parametrize("per_channel", [False, True])
def test_lambda_scan_and_adjoint_forms(B, T, D, per_channel):
    g = torch.Generator(device=DEV).manual_seed(B + T + D)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)
    u, lm, h0, w = r(B, T, D), -r(B, T, D).abs() * 3, (r(B, D), r(B, D)), r(B, T, D)
    an = r(1, 1, D).expand(B, T, D) if per_channel else r(B, T, D)
    if not per_channel:
        an[:, ::5] *= 1e5                                             # past the range of the reduction: the library's own sin and cos
    y, (hr, hi), him = ops.lambda_scan(u, lm, an, h0, keep_imag=True)
    y0, (hr0, hi0) = ops.lambda_scan(u, lm, an, h0)
    assert torch.equal(y, y0) and torch.equal(hr, hr0) and torch.equal(hi, hi0)
    ry, (rr, ri) = oracle.lambda_literal(u.double(), lm.double(), an.double(), (h0[0].double(), h0[1].double()))
    for a, b in ((y, ry), (hr, rr), (hi, ri), (him[:, -1], ri)):
        assert rel(a, b) < 5e-6
    d = ops.lambda_scan_bwd(w, u, lm, an, y, him, g_last_i=r(B, D) * 0, want_dh0=True)
    if B < 100:
        ref = oracle.lambda_scan_grads(u, lm, an, h0, w, torch.zeros(B, D, device=DEV), torch.zeros(B, D, device=DEV))
        for a, b in zip(d, ref):
            assert rel(a, b) < 2e-5


# shapes for which a pass that also writes Im h would by its own bytes be given other segments, or the other form
@pytest.mark.parametrize("B,T,D,per_channel", [
    (18, 65, 91, False), (4, 74, 305, False), (16, 88, 326, False), (21, 56, 180, False), (16, 115, 384, False),
    (22, 34, 159, True), (6, 72, 231, True), (16, 83, 158, True), (18, 53, 292, True), (11, 407, 144, True)])
def test_training_and_inference_give_the_same_bits(B, T, D, per_channel):
    g = torch.Generator(device=DEV).manual_seed(D)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)
    u, lm, h0 = r(B, T, D), -r(B, T, D).abs(), (r(B, D), r(B, D))
    an = r(1, 1, D).expand(B, T, D) if per_channel else r(B, T, D)
    y, (hr, hi), _ = ops.lambda_scan(u, lm, an, h0, keep_imag=True)
    y0, (hr0, hi0) = ops.lambda_scan(u, lm, an, h0)
    assert torch.equal(y, y0) and torch.equal(hr, hr0) and torch.equal(hi, hi0)


@pytest.mark.parametrize("B,T,D", [(2, 100, 766), (2, 1000, 766), (64, 256, 256), (3, 200, 65)])    # lanes of two channels, of four, of one
def test_the_segments_the_library_names_are_those_it_takes(B, T, D):
    g = torch.Generator(device=DEV).manual_seed(T)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)
    u, lm, an = r(B, T, D), -r(B, T, D).abs(), r(B, T, D)
    ts = _lib.lib().pgb_lambda_scan_time_segments(B, T, D, torch.cuda.get_device_properties(0).multi_processor_count)
    y, (hr, hi) = ops.lambda_scan(u, lm, an)
    y0, (hr0, hi0) = ops.lambda_scan(u, lm, an, time_segments=ts)
    assert torch.equal(y, y0) and torch.equal(hr, hr0) and torch.equal(hi, hi0)


@pytest.mark.parametrize("ts", [1, 4, 32])
@pytest.mark.parametrize("T", [2, 15, 16, 17, 33, 140, 385])
@pytest.mark.parametrize("D", [8, 68])
def test_lambda_scan_slots(ts, T, D):
    """Tiles of 4 ts steps in two slots a lane: sequences of less than one tile, of exactly one, of a few and a remainder."""
    g = torch.Generator(device=DEV).manual_seed(T + D)
    u, lm, an = (torch.randn(2, T, D, device=DEV, generator=g) for _ in range(3))
    lm = -lm.abs()
    h0 = (torch.randn(2, D, device=DEV, generator=g), torch.randn(2, D, device=DEV, generator=g))
    y, (hr, hi) = ops.lambda_scan(u, lm, an, h0, time_segments=ts)
    ry, (rr, ri) = oracle.lambda_literal(u.double(), lm.double(), an.double(), tuple(h.double() for h in h0))
    for a, b in ((y, ry), (hr, rr), (hi, ri)):
        assert rel(a, b) < 5e-6


@pytest.mark.parametrize("T", [1, 31, 32, 33, 100])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("strided", [False, True])
def test_prep_backward_row_forms(T, D, strided):
    g = torch.Generator(device=DEV).manual_seed(T)
    B, H = 2, 3
    wide = torch.randn(B, T, 3 * H * D + 8, device=DEV, generator=g).bfloat16()
    off = 4 if strided else 0                                        # 8 bytes off: the rows are not 16-byte aligned
    qp, kp, vp = (wide[..., off + i * H * D:off + (i + 1) * H * D].unflatten(-1, (H, D)) for i in range(3))
    gl = torch.randn(B, T, H, device=DEV, generator=g).bfloat16()
    th, pos = synth.rope_theta(H, D).to(DEV), 50 + torch.arange(T, device=DEV)
    dy = [torch.randn(B, H, T, D, device=DEV, generator=g).bfloat16() for _ in range(3)]
    got = ops.prep_bwd(qp, kp, vp, gl, th, pos, *dy)
    with torch.enable_grad():
        a = [t.detach().float().requires_grad_(True) for t in (qp, kp, vp, gl, th)]
        ref = torch.autograd.grad(sum((o * d.float()).sum() for o, d in zip(oracle.prep_ref(*a, pos), dy)), a)
    for x, y_, tol in zip(got, ref, (4e-3, 4e-3, 4e-3, 1e-4, 1e-3)):
        assert rel(x.float(), y_) < tol
    assert ops.prep_bwd(qp, kp, vp, gl, th, pos, *dy, want_theta=False)[4] is None


@pytest.mark.parametrize("T", [1, 63, 64, 65, 200])
@pytest.mark.parametrize("D", [64, 128])
def test_fp32_prefill_chunks(T, D):
    g = torch.Generator().manual_seed(T)
    q, k, v = (torch.nn.functional.normalize(torch.randn(2, 3, T, D, generator=g), dim=-1) for _ in range(3))
    la, S0 = -torch.rand(2, 3, T, generator=g), torch.randn(2, 3, D, D, generator=g)
    a = [t.to(DEV) for t in (q, k, v, la, S0)]
    o, S = ops.prefill(*a[:4], S0=a[4], precision=PREFILL_FP32)[:2]
    ro, rS = oracle.plain_literal(*(t.double() for t in (q, k, v, la, S0)))
    assert rel(o.cpu(), ro) < 2e-6 and rel(S.cpu(), rS) < 2e-6
