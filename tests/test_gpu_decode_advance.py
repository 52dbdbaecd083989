"""The bookkeeping between two decode steps on the device: the stand-alone launch, and the whole-step launch's own."""
import pytest
import torch

from pragnosia_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pos,window", [(0, 1), (0, 512), (510, 512), (511, 512), (1 << 40, 7)])
def test_decode_advance(pos, window):
    p, s = torch.tensor([pos], device="cuda"), torch.full((), 9.0, device="cuda")
    ops.decode_advance(p, s, window)
    assert p.item() == (pos + 1) % window and s.item() == 1.0


@pytest.mark.parametrize("token_kernel", [True, False])
def test_positions_wrap_at_the_window(token_kernel):
    from pragnosia_b200.generate import Decoder
    from pragnosia_b200.model import LM
    torch.manual_seed(0)
    with torch.device("cuda"):
        m = LM(vocab=128, d=128, layers=2, mlp_mult=2, ctx=64, mixer="aspin", norm="rms")
    d = Decoder(m.to(torch.bfloat16).eval(), batch=2, token_kernel=token_kernel)
    d.prefill(torch.randint(0, 128, (2, 62), device="cuda"))
    seen = []
    for _ in range(4):
        d.step(torch.tensor([1, 2], device="cuda"))
        seen.append((d.pos.item(), d.shift.item()))
    assert seen == [(63, 1.0), (0, 1.0), (1, 1.0), (2, 1.0)]
