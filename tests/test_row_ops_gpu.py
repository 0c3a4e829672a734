"""LayerNorm over rows that fit into registers and over longer ones, column sums over ragged sizes (csrc/jukebox.cu), against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,W", [(1, 4), (3, 1020), (2, 1024), (5, 4800), (2, 5120), (3, 5124), (1, 9000)])
def test_layernorm_of_every_width(rows, W):
    from llark_b200 import ops

    torch.manual_seed(W)
    x, g, b = torch.randn(rows, W, device="cuda") * 3 + 1, torch.randn(W, device="cuda"), torch.randn(W, device="cuda")
    want = torch.nn.functional.layer_norm(x.double(), (W,), g.double(), b.double(), 1e-5)
    # fp32 sums of up to 36 terms per thread and 8 levels: 44 * 2^-24 of the statistics, one rounding per step after them
    assert (ops.layernorm_fwd(x, g, b).double() - want).norm() <= 64 * 2.0 ** -24 * want.norm()
    assert ((ops.layernorm_fwd(x, g, b, out_dtype=torch.bfloat16).double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()


@pytest.mark.parametrize("rows,H", [(1, 1), (15, 33), (17, 64), (1000, 100), (4097, 4096)])
def test_column_sums_of_ragged_matrices(rows, H):
    from llark_b200 import ops

    torch.manual_seed(rows + H)
    x = torch.randn(rows, H, device="cuda").bfloat16()
    out = torch.randn(H, device="cuda").bfloat16()
    for acc in (False, True):
        want = x.double().sum(0) + (out.double() if acc else 0)
        got = out.clone()
        ops.colsum(x, got, accumulate=acc)
        # one rounding to eight bits, and an fp32 chain of rows / 16 + 16 terms
        bound = 2.0 ** -8 * want.abs() + (rows / 16 + 16) * 2.0 ** -24 * x.double().abs().sum(0) + 1e-6
        assert ((got.double() - want).abs() <= bound).all()
