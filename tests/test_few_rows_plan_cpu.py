"""How products with few rows are cut (csrc/skinny.cu), worked out on the host."""
import ctypes
import os

import pytest

NONE, RELU2, SILU_GLU, CLAMP_GLU = 0, 1, 4, 3


def _plan(M, N, K, act=NONE, max_tiles=0):
    from llark_b200 import _lib

    if not os.path.exists(_lib.LIB_PATH):
        pytest.skip("the library has not been built")
    out = (ctypes.c_longlong * 7)()
    assert _lib.lib().llark_few_rows_plan(M, N, K, act, max_tiles, out) == 0
    return dict(zip(("units", "rows", "cs", "box", "inner", "outer", "experts"), out))


# sizes that fill tiles of the products and sizes that do not: results of an expert, K
@pytest.mark.parametrize("ff,K", [(12, 40), (64, 64), (72, 1032), (127, 512), (768, 2048), (1024, 4096), (1000, 8)])
@pytest.mark.parametrize("act", [NONE, RELU2, SILU_GLU, CLAMP_GLU])
def test_boxes_of_routed_experts_end_with_the_experts_that_have_weights(ff, K, act):
    """Whatever max_tiles says (experts without weights are counted in it, a caller may give any upper bound): no box of an expert's tiles reaches a
    row behind the last expert's, and none misses a row of its own."""
    N = 2 * ff if act in (SILU_GLU, CLAMP_GLU) else ff
    for real, through, n_ent in ((1, 0, 1), (5, 3, 60), (8, 8, 700), (200, 1, 64)):
        for max_tiles in ((n_ent + 63) // 64 + real + through, 1, 4096):
            p = _plan(0, N, K, act, max_tiles)
            assert p["inner"] == K
            for expert in {0, real - 1}:
                seen = set()
                for u0 in range(0, ff, p["units"]):
                    first = [2 * u0] if act == CLAMP_GLU else [u0, ff + u0] if act == SILU_GLU else [u0]
                    for row in first:
                        if p["experts"]:
                            assert expert < p["experts"]
                            at = [expert * N + r for r in range(row, min(row + p["box"], p["outer"]))]
                        else:
                            at = list(range(expert * N + row, min(expert * N + row + p["box"], p["outer"])))
                        assert not at or at[-1] < real * N
                        seen.update(at)
                assert set(range(expert * N, (expert + 1) * N)) <= seen


@pytest.mark.parametrize("M", [9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("act", [NONE, SILU_GLU])
def test_chains_over_k_are_no_longer_than_those_of_whole_tiles(M, act):
    """The sums of a CTA's part of K are one chain in adders that cut instead of rounding: never longer than with tiles of 128 rows in as many CTAs
    as are resident at once (two for each of 148 SMs, clusters of up to eight, four slices of 64 or more for each)."""
    for N in (64, 1000, 1024, 2048, 2560, 3072, 4096, 4224, 4608, 6144, 8192, 12288, 22016, 32004):
        for K in (64, 504, 512, 1024, 1536, 2048, 2560, 4096, 5120, 11008):
            slices, tiles, cs = (K + 63) // 64, (N + 127) // 128, 1
            while cs < 8 and tiles * cs * 2 <= 296 and slices // (cs * 2) >= 4:
                cs *= 2
            assert -(-slices // _plan(M, N, K, act)["cs"]) <= -(-slices // cs), (N, K)
