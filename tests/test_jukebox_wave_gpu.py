"""The encoder's first convolution in the visit of the res blocks behind it (csrc/jb_chain_tc.cu): the same numbers as one after the other."""
import math
import os

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,T", [(1, 2), (2, 256), (3, 862), (1, 864), (2, 866), (1, 130002)])
@pytest.mark.parametrize("dils", [(1, 3, 9, 27), (27,), (9, 40, 1), ()])
@pytest.mark.parametrize("bad", [None, float("inf"), float("nan"), 3.4e38])
def test_the_waveform_s_convolution_in_the_blocks_visit(N, T, dils, bad):
    from llark_b200 import ops

    g = torch.Generator().manual_seed(N + T + len(dils))
    x = torch.randn(N, 1, T, generator=g)
    if bad is not None:
        x[N - 1, 0, T // 3] = x[0, 0, T - 1] = bad
    down = torch.randn(32, 1, 4, generator=g).cuda() / 2, torch.randn(32, generator=g).cuda() * 0.1
    blocks = [((torch.randn(32, 32, 3, generator=g) / math.sqrt(96)).cuda(), (torch.randn(32, generator=g) * 0.1).cuda(),
               (torch.randn(32, 32, 1, generator=g) / math.sqrt(32)).cuda(), (torch.randn(32, generator=g) * 0.1).cuda()) for _ in dils]
    x = x.cuda()
    for env in (None, "0"):
        if env:
            os.environ["LLARK_JB_CONV_TC"] = env
        try:
            got, want = ops.jb_resblocks(x, blocks, dils, down=down), ops.jb_resblocks(ops.jb_conv_down(x, *down), blocks, dils)
        finally:
            os.environ.pop("LLARK_JB_CONV_TC", None)
        assert got.shape == want.shape == (N, 32, T // 2)
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(), want.nan_to_num())
