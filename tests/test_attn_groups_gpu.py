"""Training attention where heads and samples do not fill the groups that CTAs are handed out in, query and key tiles ragged: forward and
backward against the same in 64 bits."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,NH,S,pad", [(1, 1, 1, 0), (1, 33, 129, 0), (3, 11, 300, 40), (5, 13, 64, 3), (2, 31, 640, 130)])
def test_heads_that_do_not_fill_a_group(B, NH, S, pad):
    from llark_b200 import ops

    torch.manual_seed(B * NH + S)
    H = NH * 128
    qkv = torch.randn(B * S, 3 * H, device="cuda").to(torch.bfloat16)
    dout = torch.randn(B * S, H, device="cuda").to(torch.bfloat16)
    mask = None
    if pad:
        mask = torch.ones(B, S, dtype=torch.uint8, device="cuda")
        for b in range(B):
            mask[b, S - (b * pad) // B:] = 0
    out, lse = ops.attn_fwd(qkv, mask, B, S, NH, 128)
    grad = ops.attn_bwd(qkv, mask, out, dout, lse, B, S, NH, 128)
    x = qkv.view(B, S, 3, NH, 128).double().requires_grad_(True)
    s = torch.einsum("bthd,bshd->bhts", x[:, :, 0], x[:, :, 1]) / math.sqrt(128.0)
    at = torch.arange(S, device="cuda")
    seen = (at[None] <= at[:, None])[None, None]
    if mask is not None:
        seen = seen & mask.bool()[:, None, None]
    s = s.masked_fill(~seen, -math.inf)
    want = torch.einsum("bhts,bshd->bthd", torch.softmax(s, -1), x[:, :, 2])
    g, = torch.autograd.grad(want, x, dout.view(B, S, NH, 128).double())
    rel = lambda a, b: ((a.double().view_as(b) - b).norm() / b.norm()).item()  # noqa: E731
    # probabilities, their gradients and the results in bf16: three roundings of 2^-9 at most on the way, gradients of q and k twice as many
    assert rel(out, want.detach()) < 3 * 2.0 ** -9
    assert rel(grad, g) < 6 * 2.0 ** -9
    assert torch.allclose(lse.view(B, NH, S).double(), torch.logsumexp(s.detach(), -1), atol=2e-3)
