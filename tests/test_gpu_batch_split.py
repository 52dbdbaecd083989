"""The decode linear layer with its contraction cut over a cluster (2 and 4 CTAs; whole and ragged K, residual and row sums)
against the product in fp32."""
import pytest
import torch
import torch.nn.functional as F

from pragnosia_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1024, 1032, 1536, 1608, 2048, 3072, 4104])
@pytest.mark.parametrize("N", [8, 592, 768, 1184])
@pytest.mark.parametrize("B", [1, 33, 64, 65, 128])
def test_split_contraction(K, N, B):
    g = torch.Generator(device="cuda").manual_seed(K + N + B)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, W, b, r = rn(B, K).bfloat16(), (rn(N, K) / K ** 0.5).bfloat16(), rn(N).bfloat16(), rn(B, N).bfloat16()
    lin = x.float() @ W.float().T + b.float()
    rel = lambda a, c: float((a.float() - c).norm() / c.norm())
    y = ops.batch_linear(x, W, b)
    assert rel(y, lin) < 3e-3 and torch.equal(y, ops.batch_linear(x, W, b))
    assert rel(ops.batch_linear(x, W, b, act="gelu"), F.gelu(lin)) < 4e-3
    out, sums = ops.batch_linear(x, W, b, resid=r, want_sums=True)
    assert rel(out, lin + r.float()) < 4e-3
    tot = sums.sum(0)
    assert torch.allclose(tot[:, 0], out.float().sum(1), rtol=1e-3, atol=0.05) and torch.allclose(tot[:, 1], out.float().pow(2).sum(1), rtol=1e-3)
