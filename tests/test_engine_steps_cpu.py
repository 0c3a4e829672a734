"""The step of a layer-list engine on the host: what it refuses, and that a refused step leaves the caches as they were. The layers are
stand-ins; the step descriptor and the caches are the product's."""
import types

import pytest
import torch


def _engine():
    from llark_b200.engine_seq import LayerListEngine
    from llark_b200.state_cache import StateCache

    class Rows(LayerListEngine):
        """Logits = the token at the wanted place, and its row."""
        cfg, device = types.SimpleNamespace(vocab=50), torch.device("cpu")

        def _embed(self, ids, st):
            return torch.stack([ids.float(), torch.arange(st.n_tok).float()], 1)

        def _run_layers(self, cache, x, st, residuals):
            return x

        def _logits(self, x, rows):
            return x[rows.long()]

    cache = StateCache("cpu", n_slots=3)
    cache.add_store((2,), torch.float32, True)
    return Rows(), cache, [cache.alloc(), cache.alloc()]


def test_wanted_places_in_the_order_of_the_requests():
    eng, cache, slots = _engine()
    out = eng.step(cache, slots, [[3, 4, 5], [6, 7]], want=[[2, 0], [1]])
    assert out.tolist() == [[5.0, 2.0], [3.0, 0.0], [7.0, 4.0]]
    assert eng.step(cache, slots, [[8], [9]], want=[[0]]).tolist() == [[8.0, 0.0]]
    assert eng.step(cache, slots, [[8], [9]], want=[[], [0], []]).tolist() == [[9.0, 1.0]]


@pytest.mark.parametrize("want,error", [([[0], [0], [0]], IndexError), ([[3], [0]], ValueError), ([[0], [-1]], ValueError)])
def test_wanted_places_outside_the_step_are_refused(want, error):
    eng, cache, slots = _engine()
    with pytest.raises(error):
        eng.step(cache, slots, [[3, 4, 5], [6, 7]], want=want)
    assert [cache.length[s] for s in slots] == [0, 0]


@pytest.mark.parametrize("lens,most", [([16], 1), ([1, 17, 40], 100), ([2048] + [1] * 31, 64), ([200, 70, 3, 64], 5), ([5] * 40 + [300], 8)])
def test_passes_of_the_block_walk(lens, most):
    """Every block of 16 tokens once, and no more at a time than asked for (one per request at least)."""
    from llark_b200 import ops
    from llark_b200.state_cache import StepLayout

    st = StepLayout(lens, [0] * len(lens), list(range(len(lens))), "cpu")
    left, at = [-(-n // 16) for n in lens], 0
    passes = ops.scan_passes(st.cu_host, most)
    for done, each, n, m in passes:
        take = [min(x, each) for x in left]
        assert (done, n, m) == (at, sum(x > 0 for x in left), sum(take)) and n > 0
        assert m <= max(most, n) and (each == max(left) or sum(min(x, each + 1) for x in left) > most)
        left, at = [x - t for x, t in zip(left, take)], at + each
    assert not any(left)
    if lens[0] == 2048:  # one long prompt beside single tokens: not a pass per block of it
        assert len(passes) <= 3


@pytest.mark.parametrize("H,lens,kinds", [
    (16, [16], {"scalar": False, "channel": False, "hgrn2": False}), (16, [24], {"hgrn2": True, "channel": False}),
    (32, [64], {"hgrn2": True, "channel": True, "scalar": True, "state": True}),
    (32, [32] + [1] * 31, {"hgrn2": False, "channel": False, "state": True}), (32, [64] + [1] * 127, {"hgrn2": False}),
    (32, [16] * 32, {"hgrn2": True, "channel": True, "scalar": True}), (32, [2048] + [1] * 127, {"hgrn2": True, "channel": True, "scalar": True})])
def test_the_walk_is_taken_where_it_was_faster(H, lens, kinds):
    from llark_b200 import ops

    for kind, want in kinds.items():
        assert ops.walk_pays(kind, H, max(lens), len(lens), sum(lens), sum(-(-n // 16) for n in lens)) == want, kind


def test_fp32_mode_asks_every_recurrence_for_fp32():
    """dtype=torch.float32 means no TF32: each scan that has a form on the tensor cores is told."""
    import ast
    import os

    from llark_b200 import mixers

    calls = [n for n in ast.walk(ast.parse(open(os.path.abspath(mixers.__file__)).read())) if isinstance(n, ast.Call)
             and getattr(n.func, "attr", "") in ("seq_glr_scan", "seq_delta_rule", "seq_decay_scan")]
    assert len(calls) == 5
    for c in calls:
        assert [ast.unparse(k.value) for k in c.keywords if k.arg == "full_fp32"] == ["self.act == F32"], ast.unparse(c)


def test_ops_import_on_a_torch_without_cuda():
    """The host side (layouts, passes, checks) is used and tested where torch has no CUDA; only a call needs the device."""
    import os
    import subprocess
    import sys

    code = ("import torch\n"
            "for n in ('_cuda_getCurrentRawStream', '_cuda_getDevice'):\n"
            "    if hasattr(torch._C, n): delattr(torch._C, n)\n"
            "import llark_b200.ops as ops\n"
            "assert ops.scan_passes([0, 5, 40], 4)\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-1000:]
