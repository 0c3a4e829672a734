"""The integers of a packed step: written by a launch (up to 256, 1024 and 8000 of them) or copied, the same as on the CPU; and the library's
entry points as native functions against their ctypes forms."""
import os
import random
import re

import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("n_seq,longest,extra", [(1, 1, 0), (63, 1, 0), (63, 7, 1), (3, 700, 241), (255, 3, 5), (40, 90, 863), (1999, 2, 3), (2000, 2, 0), (5, 4000, 9000)])
def test_a_step_s_integers_are_those_of_the_cpu(n_seq, longest, extra):
    from llark_b200.state_cache import StepLayout

    rng = random.Random(n_seq + extra)
    lens = [rng.randint(1, longest) for _ in range(n_seq)]
    pos, slots = [rng.randint(0, 5000) for _ in lens], rng.sample(range(4 * n_seq), n_seq)
    more = ([rng.randint(-2 ** 31, 2 ** 31 - 1) for _ in range(extra)], list(range(3)))
    want, got = StepLayout(lens, pos, slots, "cpu", more), StepLayout(lens, pos, slots, "cuda", more)
    for name in ("tok_seq", "cu", "pos0", "slot", "lens_dev"):
        assert torch.equal(getattr(got, name).cpu(), getattr(want, name)), name
    assert [e.tolist() for e in got.extra] == [list(e) for e in more] and got.max_len == want.max_len


def test_native_calls_take_what_ctypes_takes():
    from llark_b200 import _lib

    if not os.path.exists(_lib.LIB_PATH):
        pytest.skip("the library has not been built")
    native = pytest.importorskip("llark_b200._calls")
    c, n = _lib.lib(), _lib.calls()
    hdr = open(os.path.join(os.path.dirname(__file__), "..", "include", "llark_b200.h")).read()
    hdr = re.sub(r"/\*.*?\*/", " ", hdr, flags=re.S)
    launching = {m[0] for m in re.findall(r"\b(llark_\w+)\s*\(([^)]*)\)", hdr) if "cudaStream_t" in m[1]} - {"llark_grad_bucket_allreduce"}
    assert launching <= set(native.bind(os.path.abspath(c._name)))
    buf = (_lib.ctypes.c_float * 4)()
    for args in ((16, 24, 16, 24, 16, 24, 1, None, 0, 24, 24, 0, 0, 0.0, 1.702, None), (buf, 24, 16, True, 2 ** 63, -1, 1, buf, 0, 24, 24, 0, 0, 0, 2, None)):
        assert n.llark_linear_rows(*args) == -1  # no rows: refused before anything is read
    assert n.llark_seq_chunk_block_bytes(128, 1) == c.llark_seq_chunk_block_bytes(128, 1)
    for bad in ((1.5,) + (0,) * 15, (0, 1.5) + (0,) * 14, (0,) * 13 + ("x", 0, 0), (0,) * 15, (torch.zeros(1),) + (0,) * 15):
        with pytest.raises(TypeError):
            n.llark_linear_rows(*bad)


def test_native_calls_take_no_host_array_for_a_pointer():
    """What ctypes refuses for an address (an array of the host would reach a kernel as one) is refused; its own arrays and pointers are taken."""
    import array
    import ctypes

    import numpy as np

    from llark_b200 import _lib

    if not os.path.exists(_lib.LIB_PATH):
        pytest.skip("the library has not been built")
    native = pytest.importorskip("llark_b200._calls")
    _lib.calls()
    host = np.array([1, 3, 9], dtype=np.int32)
    own = (ctypes.c_int * 3)(1, 3, 9)
    for bad in (host, host[0], host.tobytes(), bytearray(12), memoryview(own), array.array("i", [1, 3, 9]), "1", ctypes.c_int(1), ctypes.byref(own), object()):
        with pytest.raises(TypeError):
            native.llark_jb_resblocks_length(bad, 3)
    want = _lib.lib().llark_jb_resblocks_length(own, 3)
    assert want == 3
    for good in (own, host.ctypes.data, ctypes.cast(own, ctypes.c_void_p), ctypes.cast(own, ctypes.POINTER(ctypes.c_int))):
        assert native.llark_jb_resblocks_length(good, 3) == want
